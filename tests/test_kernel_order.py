"""Orders that the tensor-memory and tensor-map kernels rest on, read from the
sources: a wrong one need not show in a run, and where it does the GPU hangs."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "asetsmatlabmaxflow_gb300" / "csrc"


def _body(text, start):
    """The braces' contents after position `start`."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces")


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def _kernels(name):
    text = _code(name)
    for m in re.finditer(r"__global__", text):
        k = re.compile(r"(\w+)\s*\(const __grid_constant__").search(text, m.end())
        if k and "__global__" not in text[m.end():k.start()]:
            yield k.group(1), _body(text, k.end())


@pytest.mark.parametrize("name,kernel", [("conv_tc.cu", "conv3_tc_kernel"), ("wgrad_tc.cuh", "wgrad_tc_kernel")])
def test_dependents_start_after_the_tensor_memory_is_held(name, kernel):
    """A dependent block keeps its tensor memory while it waits for this
    launch: no block of this launch may still have to allocate by then."""
    body = dict(_kernels(name))[kernel]
    alloc = body.index("tmem_alloc(")
    for m in re.finditer(r"grid_launch_dependents\(\)", body):
        assert m.start() > alloc
        # by the allocating warp itself, or after a barrier of the block
        between = body[alloc:m.start()]
        assert "}" not in between or "__syncthreads()" in between


@pytest.mark.parametrize("name", ["stencil2_kernel.cuh", "stencil2d_t2.cuh", "stencil3d_kernel.cuh"])
def test_tensor_maps_are_acquired_before_the_first_load(name):
    text = _code(name)
    found = 0
    for kernel, body in _kernels(name):
        if "issue_load" not in body:
            continue
        found += 1
        head = body[:body.index("issue_load")]
        at = re.search(r"if \(producer_warp && it >= 0\)\s*tensormaps_acquire<", head)
        assert at, kernel
        # a barrier between the warp's fences and the producer's loads
        assert "__syncthreads()" in head[at.end():], kernel
        maps = re.findall(r"(\S+)\.(?:halo|tile)\[", body)
        assert maps and all(m.endswith("P)") for m in maps) and "tensormaps(B, P)" in body, kernel
    assert found


def test_one_problem_kernels_load_through_the_launchs_maps():
    """The multi-label 2D kernels acquire nothing: every map they use is among
    their launch's parameters."""
    text = _code("stencil2d_labels.cuh")
    assert re.findall(r"lab2_issue<MODEL, L>\([^;]*", text)
    assert all(" B.maps, par" in c for c in re.findall(r"lab2_issue<MODEL, L>\([^;]*", text))
    assert set(re.findall(r"(\w+)\.(?:halo|tile)\[", text)) == {"M"}


def test_no_kernel_writes_tensor_maps():
    """Launches over one problem have their maps among their parameters; the
    kernel that writes the rest of a descriptor leaves those in it alone."""
    text = _code("init_kernels.cu")
    body = _body(text, text.index("prepare_kernel(const"))
    assert "int i = sizeof(TensorMaps) / 4 + threadIdx.x" in body and "A.d_desc)[i]" in body


@pytest.mark.parametrize("name,launches", [("runtime.cu", 2), ("noalloc.cu", 1), ("mtwin.cu", 1)])
def test_launches_say_where_their_maps_are(name, launches):
    text = _code(name)
    own, shared = text.count(".use_maps("), text.count(".own_maps = 0;")
    assert own == launches and own + shared == text.count(".total_items = ")
