"""GPU tests of calls captured into CUDA graphs: what a capture may be the first to
need, and what kind of graph comes of it.  The reference launches on the legacy
stream only (src/sgemm.cuh:33-45), which cannot be captured.
"""
import os
import subprocess
import sys

import pytest

import sgemm_b200 as sg

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# A process whose only call outside capture is a small one that needs no scratch,
# then a captured one that does.
FIRST_SCRATCH = """
import sys
sys.path[:0] = [{root!r} + "/sgemm.cu_b200"]
import torch
import sgemm_b200 as sg
path, size, pad = {path!r}, {size}, {pad}
small = [torch.rand(64, 64, device="cuda") for _ in range(3)]
sg.gemm(path, *small)
A, B, C = (torch.rand(size, size + pad, device="cuda")[:, :size] for _ in range(3))
torch.cuda.synchronize()
s = torch.cuda.Stream()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=s):
    sg.gemm(path, A, B, C, 1.0, 0.0, stream=s)
C.zero_()
g.replay()
torch.cuda.synchronize()
want = torch.empty_like(C)
sg.gemm(path, A, B, want, 1.0, 0.0)
torch.cuda.synchronize()
assert sg.device_status() == sg.OK
assert torch.equal(C, want)
print("captured")
"""


@pytest.mark.parametrize("path,size,pad", [("plain", 2048, 0), ("plain", 2001, 0),
                                           ("plain", 2048, 1), ("bf16x6", 4096, 0),
                                           ("tf32x3", 1000, 1)])
def test_first_call_with_scratch_may_be_captured(path, size, pad):
    r = subprocess.run([sys.executable, "-c",
                        FIRST_SCRATCH.format(root=ROOT, path=path, size=size, pad=pad)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]


def _captured(call):
    """The graph of call(stream) captured in global mode, and its nodes' types."""
    import torch
    rt = pytest.importorskip("cuda.bindings.runtime")

    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    h = rt.cudaStream_t(s.cuda_stream)
    assert rt.cudaStreamBeginCapture(
        h, rt.cudaStreamCaptureMode.cudaStreamCaptureModeGlobal)[0] == 0
    try:
        call(s)
    finally:
        err, graph = rt.cudaStreamEndCapture(h)
    assert err == 0
    err, _, count = rt.cudaGraphGetNodes(graph)
    err, nodes, count = rt.cudaGraphGetNodes(graph, count)
    assert err == 0
    return graph, [rt.cudaGraphNodeGetType(n)[1].name for n in nodes]


@pytest.mark.parametrize("name", ["tma_128x64_w4p_t8x8_s3", "tma_128x64_w4p_t8x8_s4",
                                  "tma_28x256_w4p_t7x8_s3_rows"])
def test_large_tiles_that_read_a_in_place(name):
    """Large tiles for calls that have no scratch: one kernel, no transposed copy."""
    import torch

    A, B, C = (torch.rand(512, 512, device="cuda") for _ in range(3))
    cfg = sg.config_names().index(name)
    sg.sgemm(A, B, C, config=cfg)
    _, kinds = _captured(lambda s: sg.sgemm(A, B, C, config=cfg, stream=s))
    assert kinds == ["cudaGraphNodeTypeKernel"]


# The fallback for calls without scratch; odd rows from 512^3 on are copied instead.
@pytest.mark.parametrize("m,n,k,pad,kinds", [
    (2048, 2048, 2048, 0, ["Kernel"]), (3000, 3000, 3000, 0, ["Kernel"]),
    (300, 520, 4096, 0, ["Kernel"]), (401, 401, 401, 0, ["Kernel"]),
    (2048, 640, 1028, 1, ["Kernel", "Kernel", "MemAlloc", "MemAlloc", "MemAlloc", "MemFree"])])
def test_captured_plain_calls_need_no_memory_nodes(m, n, k, pad, kinds):
    """A captured aligned call is one kernel, so its graph can be a child graph and be
    instantiated twice; the bits are the direct call's."""
    import torch
    rt = pytest.importorskip("cuda.bindings.runtime")

    A, B, C = (torch.rand(r, c + pad, device="cuda")[:, :c] for r, c in ((m, k), (k, n), (m, n)))
    want, C0 = C.clone(), C.clone()
    sg.sgemm(A, B, want, 1.5, 0.5)
    graph, got = _captured(lambda s: sg.sgemm(A, B, C, 1.5, 0.5, stream=s))
    got = {x.replace("cudaGraphNodeType", "") for x in got}
    assert got == set(kinds)
    if kinds != ["Kernel"]:
        return
    err, parent = rt.cudaGraphCreate(0)
    assert err == 0 and rt.cudaGraphAddChildGraphNode(parent, None, 0, graph)[0] == 0
    first, second = rt.cudaGraphInstantiate(parent, 0), rt.cudaGraphInstantiate(graph, 0)
    assert first[0] == 0 and second[0] == 0
    for exe in (first[1], second[1]):
        C.copy_(C0)
        torch.cuda.synchronize()
        assert rt.cudaGraphLaunch(exe, rt.cudaStream_t(0))[0] == 0
        torch.cuda.synchronize()
        assert torch.equal(C, want)
    assert sg.device_status() == sg.OK


def test_captured_call_of_a_named_tile_needs_no_memory_nodes():
    """The same where the caller names a tile that reads A transposed."""
    import torch

    A, B, C = (torch.rand(512, 512, device="cuda") for _ in range(3))
    cfg = sg.config_names().index("tma_128x64_w4_t8x8_s3")
    sg.sgemm(A, B, C, config=cfg)
    _, kinds = _captured(lambda s: sg.sgemm(A, B, C, config=cfg, stream=s))
    assert kinds == ["cudaGraphNodeTypeKernel"]
