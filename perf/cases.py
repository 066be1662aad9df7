"""Performance cases: what a user of this package has it do, through its
public entry points, from the smallest calls to the largest.

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what the user's program has in hand before the call
  run(state)           one pass through the public entry points, with its outputs
  work(case)           bytes and operations one pass cannot do without
  exact(case, seed)    the outputs in 64 bits, in plain torch

A case is a dict of plain values; `kind` says which entry points it goes
through:

  mex      the mex interface on host arrays (solvers.py), as Matlab calls it
  solver   a resident solver fed from device arrays (native.Solver)
  batch    many uneven binary problems in one batch (native.Batch)
  matlab   the Matlab-semantics solvers on host arrays (matlab.py)
  hmf      the hierarchical max-flow classes on host arrays (hmf.py)
  inputs   cost terms and contrast weights built on the device (the C ABI)
  train    loss and gradients of the warm-start network (native.WarmStartNet)

Volumes are (labels,) nz, nx, ny C-ordered tensors: the memory layout of a
Matlab ny x nx x nz (x labels) array.
"""
import math

import numpy as np
import torch

from asetsmatlabmaxflow_gb300 import hmf, matlab, solvers
from asetsmatlabmaxflow_gb300 import native as N

CC = 0.3
STEP2, STEP3 = 0.16, 0.11


def listed():
    return [
        # The smallest call: one 256^2 image from Matlab, to convergence (the
        # reference's first configuration).
        dict(name="mex binary 256x256", kind="mex", model="binary", ny=256, nx=256, nz=1, nlab=1,
             its=300, err=1e-4, exact=False),
        # A multi-region 2D call from Matlab with odd sides.
        dict(name="mex potts 301x170 L4", kind="mex", model="potts", ny=301, nx=170, nz=1, nlab=4,
             its=300, err=1e-4, exact=False),
        # The headline: a resident binary 256^3 volume, fixed iterations.
        dict(name="solver binary 256^3", kind="solver", model="binary", ny=256, nx=256, nz=256,
             nlab=1, its=100, err=0.0, exact=False),
        # An uneven volume in the mode that reproduces the reference's bits.
        dict(name="solver binary exact 181x150x97", kind="solver", model="binary", ny=181, nx=150,
             nz=97, nlab=1, its=100, err=0.0, exact=True),
        # Multi-region segmentation of a 192^3 volume to convergence.
        dict(name="solver potts 192^3 L4", kind="solver", model="potts", ny=192, nx=192, nz=192,
             nlab=4, its=300, err=1e-4, exact=False),
        # Ordered labels on a large image.
        dict(name="solver ishikawa 1024^2 L8", kind="solver", model="ishikawa", ny=1024, nx=1024,
             nz=1, nlab=8, its=100, err=0.0, exact=False),
        # A mixed batch of images and volumes, each to its own convergence.
        dict(name="batch 12x2d 4x3d", kind="batch", n2d=12, n3d=4, lo2=128, hi2=512, lo3=48, hi3=128,
             its=300, err=1e-4),
        # The tutorials' gpuArray path in single precision on a volume.
        dict(name="matlab binary f32 160x192x144", kind="matlab", model="binary", ny=160, nx=192,
             nz=144, nlab=1, its=150, err=0.0, f64=False),
        # The same path in Matlab's default class, double, on an image.
        dict(name="matlab potts f64 512x480 L4", kind="matlab", model="potts", ny=512, nx=480, nz=1,
             nlab=4, its=150, err=0.0, f64=True),
        # A label tree of six nodes below the root on an image.
        dict(name="hmf 2d 768x640", kind="hmf", ny=768, nx=640, nz=1, its=200, f64=False),
        # The step before a four-region solve of a volume: cost terms from the
        # user's scribbles, weights from the image's contrast.
        dict(name="inputs 256x231x256 L4", kind="inputs", cost="histogram", ny=256, nx=231, nz=256,
             nlab=4),
        # Forward and backward of the warm-start network at its training size.
        dict(name="train 32^3 L6", kind="train", ny=32, nx=32, nz=32, nlab=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mex", "mex", "solver", "solver", "solver", "batch", "matlab", "matlab",
                       "hmf", "inputs", "train"])
    if kind in ("mex", "solver", "matlab"):
        model = rng.choice(["binary", "potts", "ishikawa"])
        nlab = 1 if model == "binary" else rng.randint(2 if model == "potts" else 3, 6)
        c = dict(kind=kind, model=model, nlab=nlab)
        if rng.random() < 0.5:
            hi = {"mex": 700, "solver": 1500, "matlab": 700}[kind]
            c.update(ny=_log(rng, 48, hi), nx=_log(rng, 48, hi), nz=1)
        else:
            hi = {"mex": 128, "solver": 190, "matlab": 128}[kind]
            c.update(ny=_log(rng, 24, hi), nx=_log(rng, 24, hi), nz=_log(rng, 16, hi))
        conv = kind != "matlab" and rng.random() < 0.5
        c.update(its=200 if conv else rng.randint(40, 100), err=1e-4 if conv else 0.0)
        if kind == "matlab":
            c["f64"] = rng.random() < 0.5
        else:
            c["exact"] = rng.random() < 0.3
        return c
    if kind == "batch":
        return dict(kind=kind, n2d=rng.randint(4, 16), n3d=rng.randint(1, 5), lo2=64,
                    hi2=_log(rng, 192, 640), lo3=32, hi3=_log(rng, 64, 128), its=200, err=1e-4)
    if kind == "hmf":
        c = dict(kind=kind, f64=rng.random() < 0.25, its=rng.randint(50, 150))
        if rng.random() < 0.5:
            c.update(ny=_log(rng, 64, 800), nx=_log(rng, 64, 800), nz=1)
        else:
            c.update(ny=_log(rng, 24, 80), nx=_log(rng, 24, 80), nz=_log(rng, 16, 64))
        return c
    if kind == "inputs":
        return dict(kind=kind, cost=rng.choice(["histogram", "l1", "neglog"]), ny=_log(rng, 64, 256),
                    nx=_log(rng, 64, 256), nz=rng.choice([1, _log(rng, 32, 256)]),
                    nlab=rng.randint(2, 6))
    return dict(kind="train", ny=_log(rng, 16, 48), nx=_log(rng, 16, 48), nz=_log(rng, 16, 48),
                nlab=rng.randint(3, 6))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _voronoi(g, dims, values, sigma, ncells):
    """A piecewise-constant image (nearest of ncells seeds) plus noise, in [0, 1]."""
    ny, nx, nz = dims
    y = torch.arange(ny, device="cuda", dtype=torch.float32)
    x = torch.arange(nx, device="cuda", dtype=torch.float32)[:, None]
    z = torch.arange(nz, device="cuda", dtype=torch.float32)[:, None, None]
    vals = torch.tensor(values, device="cuda", dtype=torch.float32)
    pos = _rand(g, ncells, 3) * torch.tensor([ny, nx, nz], device="cuda", dtype=torch.float32)
    pick = vals[(_rand(g, ncells) * len(values)).long().clamp_(max=len(values) - 1)]
    best = torch.full((nz, nx, ny), math.inf, device="cuda")
    img = torch.empty_like(best)
    for i in range(ncells):
        d = (y - pos[i, 0]) ** 2 + (x - pos[i, 1]) ** 2 + (z - pos[i, 2]) ** 2
        near = d < best
        img = torch.where(near, pick[i], img)
        best = torch.where(near, d, best)
    img += sigma * torch.randn(img.shape, generator=g, device="cuda")
    return img.clamp_(0, 1)


def _smooth(g, dims, sigma):
    """A smooth field in [0, 1] plus noise (ordered labels)."""
    ny, nx, nz = dims
    y = torch.arange(ny, device="cuda", dtype=torch.float32)
    x = torch.arange(nx, device="cuda", dtype=torch.float32)[:, None]
    z = torch.arange(nz, device="cuda", dtype=torch.float32)[:, None, None]
    f = torch.zeros((nz, nx, ny), device="cuda")
    for _ in range(16):
        c = _rand(g, 5)
        w = (0.05 + 0.2 * c[3]) * min(ny, nx)
        d = (y - c[0] * ny) ** 2 + (x - c[1] * nx) ** 2 + (z - c[2] * nz) ** 2
        f += (2 * c[4] - 1) * torch.exp(-d / (2 * w * w))
    f = (f - f.min()) / (f.max() - f.min())
    return f + sigma * torch.randn(f.shape, generator=g, device="cuda")


def _problem(g, model, dims, nlab):
    """(Cs, Ct, alpha): costs against region means, constant weights, or
    contrast-sensitive ones for a binary volume."""
    if model == "binary":
        vol = dims[2] > 1
        img = _voronoi(g, dims, (0.25, 0.75) if vol else (0.2, 0.8), 0.2 if vol else 0.15,
                       40 if vol else 12)
        if vol:
            g2 = sum(torch.gradient(img, dim=d)[0] ** 2 for d in range(3) if img.shape[d] > 1)
            alpha = 0.1 + 0.9 * torch.exp(-10.0 * g2)
        else:
            alpha = torch.full_like(img, 0.5)
        return (img - 0.2).abs(), (img - 0.8).abs(), alpha
    if model == "potts":
        means = [0.1 + 0.8 * k / max(nlab - 1, 1) for k in range(nlab)]
        img = _voronoi(g, dims, means, 0.1, 60)
        ct = torch.stack([(img - m).abs() for m in means])
        return None, ct, torch.full_like(ct, 0.3)
    img = _smooth(g, dims, 0.05)
    ct = torch.stack([(img - k / (nlab - 1)).abs() for k in range(nlab)])
    return None, ct, torch.full_like(ct[1:], 0.2)


def _dims(case):
    return case["ny"], case["nx"], case["nz"]


def _steps(case):
    return STEP3 if case["nz"] > 1 else STEP2


def _matlab_array(t, dims, dtype=np.float32):
    """A tensor as the Matlab array (Fortran order) a caller holds."""
    ny, nx, nz = dims
    lab = t.shape[0] if t.dim() == 4 else 1
    shape = (ny, nx) + ((nz,) if nz > 1 else ()) + ((lab,) if t.dim() == 4 else ())
    return np.asfortranarray(t.cpu().numpy().astype(dtype).ravel().reshape(shape, order="F"))


def _batch_dims(case, seed):
    r = np.random.default_rng(seed)
    out = [(int(r.integers(case["lo2"], case["hi2"] + 1)), int(r.integers(case["lo2"], case["hi2"] + 1)), 1)
           for _ in range(case["n2d"])]
    return out + [tuple(int(v) for v in r.integers(case["lo3"], case["hi3"] + 1, 3))
                  for _ in range(case["n3d"])]


def _batch_seed(case):
    """The batch's shapes belong to the case, its images to the seed."""
    return case["n2d"] * 1000003 + case["n3d"] * 10007 + case["hi2"] * 101 + case["hi3"]


def _batch_problems(case, seed):
    g = _gen(seed)
    out = []
    for dims in _batch_dims(case, _batch_seed(case)):
        cs, ct, al = _problem(g, "binary", dims, 1)
        out.append((dims, cs, ct, torch.full_like(al, 0.2 + 0.6 * float(_rand(g, 1)))))
    return out


#: The label tree of the hmf cases: two inner nodes below the root, two leaves each.
HMF_ALPHA_LEAF, HMF_ALPHA_INNER = 0.15, 0.1


def _hmf_costs(case, seed):
    dims = _dims(case)
    img = _voronoi(_gen(seed), dims, (0.1, 0.4, 0.6, 0.9), 0.1, 30)
    return torch.stack([(img - m).abs() for m in (0.1, 0.4, 0.6, 0.9)])


def _inputs(case, seed):
    g = _gen(seed)
    dims = _dims(case)
    L = case["nlab"]
    means = [0.1 + 0.8 * k / (L - 1) for k in range(L)]
    img = _voronoi(g, dims, means, 0.08, 40) * 231.0 + 12.0   # an 8-bit scanner's range
    data = img
    scrib = None
    if case["cost"] == "histogram":
        near = ((img - 12.0) / 231.0 - torch.tensor(means, device="cuda")[:, None, None, None]).abs()
        scrib = (near.argmin(0) + 1).int()
        scrib[_rand(g, *img.shape) > 0.05] = 0
    elif case["cost"] == "neglog":
        near = ((img - 12.0) / 231.0 - torch.tensor(means, device="cuda")[:, None, None, None]).abs()
        data = torch.softmax(-20.0 * near, 0).contiguous()
    return img.contiguous(), data, scrib, means


def _train(case, seed):
    g = _gen(seed)
    dims = _dims(case)
    L = case["nlab"]
    _, ct, _ = _problem(g, "potts", dims, L)
    shape = ct.shape[1:]
    alpha = torch.full(shape, 0.1 + 0.4 * float(_rand(g, 1)), device="cuda")
    u = torch.nn.functional.one_hot(ct.argmin(0), L).permute(3, 0, 1, 2).float().contiguous()
    ps = ct.amin(0).contiguous()
    pt = torch.minimum(ct, ps + 0.05).contiguous()
    flows = [(0.3 * alpha * torch.randn(ct.shape, generator=g, device="cuda")).contiguous()
             for _ in range(3)]
    params = torch.randn(N.WarmStartNet.num_params(), generator=g, device="cuda").cpu().numpy()
    return ct.contiguous(), alpha, u, ps, pt, flows, (0.06 * params).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    ctx = N.Context.default()
    if kind == "mex":
        dims = _dims(case)
        cs, ct, al = _problem(_gen(seed), case["model"], dims, case["nlab"])
        name = {"binary": "BinaryMF", "potts": "Potts", "ishikawa": "Ishikawa"}[case["model"]]
        st["fn"] = getattr(solvers, "asets%s%dD_mex" % (name, 3 if case["nz"] > 1 else 2))
        args = [_matlab_array(t, dims) for t in (cs, ct, al) if t is not None]
        pars = [case["ny"], case["nx"]] + ([case["nz"]] if case["nz"] > 1 else [])
        pars += [] if case["model"] == "binary" else [case["nlab"]]
        pars += [case["its"], case["err"], CC, _steps(case)]
        st["args"] = args + [np.array(pars, np.float32)]
    elif kind == "solver":
        dims = _dims(case)
        cs, ct, al = _problem(_gen(seed), case["model"], dims, case["nlab"])
        st["in"] = [t if t is None else t.contiguous() for t in (ct, al, cs)]
        st["solver"] = N.Solver(ctx, case["model"], dims if case["nz"] > 1 else dims[:2], case["nlab"])
        st["u"] = torch.empty(st["solver"].n * st["solver"].u_labels, device="cuda")
    elif kind == "batch":
        st["in"], st["solvers"], st["u"] = [], [], []
        st["batch"] = N.Batch(ctx)
        for dims, cs, ct, al in _batch_problems(case, seed):
            s = N.Solver(ctx, "binary", dims if dims[2] > 1 else dims[:2])
            st["batch"].add(s)
            st["solvers"].append(s)
            st["in"].append((ct, al, cs))
            st["u"].append(torch.empty(s.n, device="cuda"))
    elif kind == "matlab":
        dims = _dims(case)
        cs, ct, al = _problem(_gen(seed), case["model"], dims, case["nlab"])
        dt = np.float64 if case["f64"] else np.float32
        name = {"binary": "BinaryMF", "potts": "Potts", "ishikawa": "Ishikawa"}[case["model"]]
        st["fn"] = getattr(matlab, "asets%s%dD" % (name, 3 if case["nz"] > 1 else 2))
        pars = [case["ny"], case["nx"]] + ([case["nz"]] if case["nz"] > 1 else [])
        pars += [] if case["model"] == "binary" else [case["nlab"]]
        pars += [case["its"], case["err"], CC, _steps(case)]
        st["args"] = [_matlab_array(t, dims, dt) for t in (cs, ct, al) if t is not None] + [pars]
    elif kind == "hmf":
        dt = np.float64 if case["f64"] else np.float32
        cls = hmf.asetsHMF3D if case["nz"] > 1 else hmf.asetsHMF2D
        leaves = [cls([], HMF_ALPHA_LEAF, _matlab_array(c, _dims(case), dt))
                  for c in _hmf_costs(case, seed)]
        inner = [cls(leaves[:2], HMF_ALPHA_INNER), cls(leaves[2:], HMF_ALPHA_INNER)]
        st["root"], st["nodes"] = cls(inner, 0), leaves + inner
    elif kind == "inputs":
        st["img"], st["data"], st["scrib"], means = _inputs(case, seed)
        st["models"] = np.array(means, np.float32)
        st["ctx"] = ctx.handle
        L = case["nlab"]
        st["ct"] = torch.empty((L,) + st["img"].shape, device="cuda")
        st["alpha"] = torch.empty((L,) + st["img"].shape, device="cuda")
        st["hist"] = np.zeros((L, 256), np.uint32)
    else:
        st["in"] = _train(case, seed)
        st["net"] = N.WarmStartNet(ctx, case["nlab"])
        st["net"].set_params(st["in"][6])
    torch.cuda.synchronize()  # the package's stream does not wait for torch's
    return st


# ---------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "mex":
        u, err, it, _ = st["fn"](*st["args"], exact=case["exact"])
        return u, err, int(it[0, 0])
    if kind == "solver":
        s = st["solver"]
        ct, al, cs = st["in"]
        s.set_inputs(ct, al, cs, where=N.DEVICE)
        it = s.run(case["its"], case["err"], CC, _steps(case), exact=case["exact"])
        s.get_u(st["u"], where=N.DEVICE)
        return st["u"], s.get_cvg(), it
    if kind == "batch":
        for s, i in zip(st["solvers"], st["in"]):
            s.set_inputs(*i, where=N.DEVICE)
        its = st["batch"].run(case["its"], case["err"], CC, STEP3)
        for s, u in zip(st["solvers"], st["u"]):
            s.get_u(u, where=N.DEVICE)
        return st["u"], its
    if kind == "matlab":
        u, err, it, _ = st["fn"](*st["args"])
        return u, err, it
    if kind == "hmf":
        root = st["root"]
        root.MaxFullFlow(case["its"], 0.1, 0.25)
        return [n.u for n in st["nodes"]], [n.pt for n in st["nodes"]], root.dataCost, root.reguCost
    if kind == "inputs":
        L, lib, img = case["nlab"], N.lib(), st["img"]
        ct, n = st["ct"].data_ptr(), st["img"].numel()
        if case["cost"] == "histogram":
            N.check(lib.asets_cost_histogram_ll(st["ctx"], N.DEVICE, img.data_ptr(),
                                                st["scrib"].data_ptr(), n, L, 1e-10, ct,
                                                st["hist"].ctypes.data))
        elif case["cost"] == "l1":
            N.check(lib.asets_cost_l1(st["ctx"], N.DEVICE, img.data_ptr(), n, st["models"].ctypes.data,
                                      L, 1, ct))
        else:
            N.check(lib.asets_cost_neglog(st["ctx"], N.DEVICE, st["data"].data_ptr(), n, L, 1e-10, ct))
        N.check(lib.asets_alpha_contrast(st["ctx"], N.DEVICE, img.data_ptr(), *_dims(case), 1, 0.05,
                                         0.3, 10.0, 0, L, st["alpha"].data_ptr()))
        return st["ct"], st["alpha"], st["hist"].astype(np.int64)
    ct, al, u, ps, pt, fl, _ = st["in"]
    loss, grads = st["net"].gradients(_dims(case), ct, al, u, ps, pt, *fl)
    return loss, grads


# ---------------------------------------------------------------- work
def _solve_work(model, voxels, nlab, three, its, size):
    """Inputs once, outputs once, and per iteration the state read and
    written once (flows, sink and source flows, multipliers; the inputs are
    read again, as none of it fits on the chip at size)."""
    flows = nlab - 1 if model == "ishikawa" else nlab
    axes = 3 if three else 2
    state = flows * (axes + 1) + {"binary": 2, "potts": nlab + 1, "ishikawa": nlab}[model]
    inputs = {"binary": 3, "potts": 2 * nlab, "ishikawa": 2 * nlab - 1}[model]
    words = inputs + flows + its * (2 * state + inputs)
    return size * voxels * words, its * voxels * flows * (20 * axes + 20)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        for ny, nx, nz in _batch_dims(case, _batch_seed(case)):
            x, y = _solve_work("binary", ny * nx * nz, 1, nz > 1, 20, 4)   # a typical count to 1e-4
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    n = case["ny"] * case["nx"] * case["nz"]
    L = case["nlab"] if "nlab" in case else 1
    if kind in ("mex", "solver", "matlab"):
        its = case["its"] if case["err"] == 0 else {"binary": 12, "potts": 45, "ishikawa": 70}[case["model"]]
        b, f = _solve_work(case["model"], n, L, case["nz"] > 1, its, 8 if case.get("f64") else 4)
    elif kind == "hmf":
        size, axes = (8 if case["f64"] else 4), (3 if case["nz"] > 1 else 2)
        words = 4 + 12 + case["its"] * (4 + 2 * (6 * (axes + 2) + 1))
        b, f = size * n * words, case["its"] * n * 6 * (20 * axes + 20)
    elif kind == "inputs":
        reads = {"histogram": 2, "l1": 1, "neglog": L + 1}[case["cost"]]
        b, f = 4 * n * (reads + 2 * L), n * (30 + 2 * L)
    else:
        b = 4 * n * (6 * L + 2 + 5 * L + 1) + 2 * 4 * N.WarmStartNet.num_params()
        f = n * 27 * 256 * 2 * (5 + 5 + 4)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- 64 bits
def _lo(t, ax):
    return t.narrow(ax, 0, t.shape[ax] - 1)


def _hi(t, ax):
    return t.narrow(ax, 1, t.shape[ax] - 1)


def _project64(b, step_src, alpha, axes, half):
    """Gradient step from step_src, projection onto |p| <= alpha, rescale, in
    place on the lower-face flows b; returns the divergence."""
    for f, ax in zip(b, axes):
        _hi(f, ax).add_(torch.diff(step_src, dim=ax))
    s = torch.zeros_like(b[0])
    for f, ax in zip(b, axes):
        s += f * f
        _lo(s, ax).add_(_hi(f, ax) ** 2)
    norm = torch.sqrt(s * 0.5 if half else s)
    gk = torch.where(norm <= alpha, 1.0, alpha / norm)
    div = torch.zeros_like(b[0])
    for f, ax in zip(b, axes):
        _hi(f, ax).mul_(0.5 * (_lo(gk, ax) + _hi(gk, ax)))
        div -= f
        _lo(div, ax).add_(_hi(f, ax))
    return div


def _solve64(model, cs, ct, alpha, three, its, err, cc, steps, twin):
    """The solvers' iteration; `twin`: the Matlab twins' initial state, `<`
    and denominator.  Returns (u, erriter)."""
    axes = [-3, -2, -1] if three else [-2, -1]
    cs = None if cs is None else cs.double()
    ct, alpha = ct.double(), alpha.double()
    if model == "binary":
        u = (cs - ct >= 0).double()
        ps = torch.minimum(cs, ct)
        pt = ps.clone()
    else:
        L = ct.shape[0]
        m, arg = ct.min(0)
        ids = torch.arange(L, device=ct.device)[:, None, None, None]
        pt = m[None].repeat(L, 1, 1, 1)
        if model == "potts":
            ps, u = m, (ids == arg[None]).double()
        else:
            u = (ids[:-1] < arg[None]).double()
            if not twin:
                pt[-1] = 0
    b = [torch.zeros_like(u) for _ in axes]
    div = torch.zeros_like(u)
    cvg = np.zeros(max(its, 1))
    denom = u.numel() if model != "ishikawa" or not twin else ct.numel() - 1
    for i in range(its):
        if model == "ishikawa":
            src = div - ((pt[:-1] - pt[1:]) + u / cc)
        else:
            src = div - ((ps - pt) + u / cc)
        div = _project64(b, steps * src, alpha, axes, True)
        if model == "binary":
            ps = torch.minimum(pt - u / cc + div + 1 / cc, cs)
            pt = torch.minimum(ps + u / cc - div, ct)
            e = cc * (pt + div - ps)
        elif model == "potts":
            pt = torch.minimum(ps + u / cc - div, ct)
            ps = (div + pt - u / cc).sum(0) / L + 1 / (cc * L)
            e = cc * (div + pt - ps)
        else:
            for k in range(L):
                up = (div[k] + pt[k + 1] - u[k] / cc) if k < L - 1 else 0
                down = (-div[k - 1] + pt[k - 1] + u[k - 1] / cc) if k else 1 / cc
                v = up + down
                pt[k] = torch.minimum(v / 2 if 0 < k < L - 1 else v, ct[k])
            e = cc * (div + pt[1:] - pt[:-1])
        u = u - e
        cvg[i] = float(e.abs().sum()) / denom
        lt = twin or (model == "ishikawa" and not three)
        if cvg[i] < err or (not lt and cvg[i] <= err):
            break
    return u, cvg


def _as_matlab(u, dims, labelled):
    """A (labels,) nz, nx, ny tensor as the ny x nx (x nz)(x labels) array."""
    ny, nx, nz = dims
    shape = (ny, nx) + ((nz,) if nz > 1 else ()) + ((u.shape[0],) if labelled else ())
    return u.cpu().numpy().ravel().reshape(shape, order="F")


def _hmf64(case, seed):
    ct = _hmf_costs(case, seed).double()
    t = np.float64 if case["f64"] else np.float32
    cc, steps = float(t(0.25)), float(t(0.1))
    axes = [-3, -2, -1] if case["nz"] > 1 else [-2, -1]
    parent = [4, 4, 5, 5, None, None]   # leaves 0-3, inner nodes 4, 5; None: the root
    al = torch.tensor([float(t(HMF_ALPHA_LEAF))] * 4 + [float(t(HMF_ALPHA_INNER))] * 2,
                      device="cuda", dtype=torch.float64)[:, None, None, None]
    shape = (6,) + tuple(ct.shape[1:])
    u, pt, div = (torch.zeros(shape, device="cuda", dtype=torch.float64) for _ in range(3))
    b = [torch.zeros_like(u) for _ in axes]
    root = torch.zeros_like(ct[0])
    for _ in range(case["its"]):
        above = lambda i: root if parent[i] is None else pt[parent[i]]  # noqa: E731
        old = [above(i).clone() for i in range(6)]
        for i in range(4):
            pt[i] = torch.minimum(ct[i], old[i] - div[i] + u[i] / cc)
        for i in (4, 5):
            kids = [k for k in range(4) if parent[k] == i]
            v = old[i] - div[i] + u[i] / cc + sum(pt[k] + div[k] - u[k] / cc for k in kids)
            pt[i] = v / (1 + len(kids))
        root = (1 / cc + sum(pt[k] + div[k] - u[k] / cc for k in (4, 5))) / 2
        for i in range(6):
            u[i] += cc * (above(i) - div[i] - pt[i])
        src = torch.stack([div[i] + pt[i] - above(i) - u[i] / cc for i in range(6)])
        div = _project64(b, steps * src, al, axes, False)
    us = [_as_matlab(u[i], _dims(case), False) for i in range(6)]
    pts = [_as_matlab(pt[i], _dims(case), False) for i in range(6)]
    return us, pts, float((u[:4] * ct).sum()), float((u * div).sum())


def _inputs64(case, seed):
    img, data, scrib, means = _inputs(case, seed)
    x = img.double()
    x = (x - x.min()) / (x.max() - x.min())
    g2 = sum(torch.gradient(x, dim=d)[0] ** 2 for d in range(3) if x.shape[d] > 1)
    alpha = float(np.float32(0.05)) + float(np.float32(0.3)) * torch.exp(-10.0 * torch.sqrt(g2))
    if case["cost"] == "l1":
        ct = torch.stack([(x - float(np.float32(m))).abs() for m in means])
    elif case["cost"] == "neglog":
        ct = -torch.log(data.double() + 1e-10)
    else:
        # the bin of a voxel is a whole number formed in single precision
        f = (img - img.min()) / (img.max() - img.min()) * 255.0
        low = f.floor().long().clamp_(0, 255)
        near = torch.floor(f.double() + 0.5).long().clamp_(0, 255)
        tabs = []
        for l in range(case["nlab"]):
            h = torch.bincount(low[scrib == l + 1], minlength=256).double()
            tabs.append(-torch.log10(h / h.sum() + 1e-10))
        ct = torch.stack([t[near] for t in tabs])
    return ct, alpha[None].expand(case["nlab"], -1, -1, -1).contiguous(), None


def _train64(case, seed):
    ct, alpha, u, ps, pt, fl, params = _train(case, seed)
    L, nw = case["nlab"], 27 * 256
    p = torch.tensor(params, device="cuda", dtype=torch.float64, requires_grad=True)

    def conv(x, b):
        w = p[b * (nw + 16):b * (nw + 16) + nw].view(3, 3, 3, 16, 16).permute(4, 3, 0, 1, 2)
        return torch.nn.functional.conv3d(x, w, p[b * (nw + 16) + nw:(b + 1) * (nw + 16)], padding=1)

    x = torch.zeros((1, 16) + tuple(alpha.shape), device="cuda", dtype=torch.float64)
    x[0, :L], x[0, L] = ct, alpha
    for b in range(3):
        x = conv(x, b).relu()
    out = torch.cat([conv(x, 3), conv(x, 4)], 1)[0, :5 * L + 1]
    target = torch.cat([u, ps[None], pt] + [f / alpha for f in fl]).double()
    loss = ((out - target) ** 2).mean()
    loss.backward()
    return float(loss.detach()), p.grad


def exact(case, seed):
    kind = case["kind"]
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    if kind in ("mex", "solver", "matlab"):
        cs, ct, al = _problem(_gen(seed), case["model"], _dims(case), case["nlab"])
        num = float if kind == "matlab" and case["f64"] else f32
        u, cvg = _solve64(case["model"], cs, ct, al, case["nz"] > 1, case["its"], num(case["err"]),
                          num(CC), num(_steps(case)), kind == "matlab")
        if kind == "solver":
            return u.reshape(-1), cvg, None
        return _as_matlab(u, _dims(case), case["model"] != "binary"), cvg.reshape(-1, 1), None
    if kind == "batch":
        us = [_solve64("binary", cs, ct, al, dims[2] > 1, case["its"], f32(case["err"]), f32(CC),
                       f32(STEP3), False)[0].reshape(-1)
              for dims, cs, ct, al in _batch_problems(case, seed)]
        return us, [None] * len(us)
    if kind == "hmf":
        return _hmf64(case, seed)
    if kind == "inputs":
        return _inputs64(case, seed)
    return _train64(case, seed)
