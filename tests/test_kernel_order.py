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


@pytest.mark.parametrize("name", ["stencil2_kernel.cuh", "stencil2d_t2.cuh", "stencil2d_labels.cuh",
                                  "stencil3d_kernel.cuh"])
def test_tensor_maps_are_acquired_before_the_first_load(name):
    text = _code(name)
    found = 0
    for kernel, body in _kernels(name):
        if "issue_load" not in body:
            continue
        found += 1
        head = body[:body.index("issue_load")]
        if "lab2_next_item(" in head:
            head = _body(text, text.index("bool lab2_next_item("))
        at = re.search(r"if \(producer_warp && it >= 0\)\s*tensormaps_acquire<", head)
        assert at, kernel
        # a barrier between the warp's fences and the producer's loads
        assert "__syncthreads()" in head[at.end():], kernel
    assert found


def test_tensor_maps_written_by_a_kernel_are_released():
    text = _code("init_kernels.cu")
    body = _body(text, text.index("prepare_kernel(const"))
    assert body.index("tensormap_release()") > body.index("A.d_desc)[i]")
