"""Kernels whose set-up overlaps the end of the kernel before them (programmatic dependent launch): what it must not cost."""
import ctypes
import re
import sys
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent
PKG_DIR = ROOT / "ascend-python_b200"


@pytest.fixture(scope="module")
def npu():
    sys.path.insert(0, str(PKG_DIR))
    try:
        import torch_npu
    finally:
        sys.path.pop(0)
    return torch_npu


def _us(calls, n=40):
    """Device time of one round of `calls`, best of five measurements of n rounds queued behind a spinning kernel."""
    for f in calls:
        f()
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(4_000_000)
        a.record()
        for _ in range(n):
            for f in calls:
                f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / n)
    return best


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["quant", "rms", "rms_quant", "matmul"])
def test_odd_columns_back_to_back(npu, dev, op):
    """Kernels of a few long-running CTAs for every SM (rows and outputs of odd widths), repeated calls: no slower than with
    a kernel of one element in between, which keeps the launches from overlapping."""
    x = torch.randn((300, 16383), device=dev, dtype=torch.bfloat16)
    gamma = torch.rand(16383, device=dev).to(torch.bfloat16)
    a = torch.ones((600, 4096), dtype=torch.int8, device=dev)
    w = torch.ones((4096, 1001), dtype=torch.int8, device=dev)
    scale = torch.rand(1001, device=dev)
    one = torch.zeros(1, device=dev)
    call = {"quant": lambda: npu.npu_dynamic_quant(x), "rms": lambda: npu.npu_rms_norm(x, gamma),
            "rms_quant": lambda: npu.npu_rms_norm_dynamic_quant(x, gamma),
            "matmul": lambda: npu.npu_quant_matmul(a, w, scale, output_dtype=torch.bfloat16)}[op]
    together, apart = _us([call]), _us([call, lambda: one.add_(1)])
    assert together < apart, f"{together:.1f} us back to back, {apart:.1f} us apart"


def test_released_behind_the_tensor_memory_allocation():
    """A kernel that allocates tensor memory releases its successor behind that, in the allocating warp: released earlier,
    a CTA of another kernel could hold the columns and wait for this one.  Read from the sources."""
    checked = 0
    for f in sorted((PKG_DIR / "csrc").glob("*.[ci]*")):
        for body in re.split(r"\b__global__\b", re.sub(r"//[^\n]*", "", f.read_text()))[1:]:
            if "tmem_alloc" in body and "pdl_launch_dependents" in body:
                block = re.search(r"if \(warp == \w+\) \{\s*tmem_alloc[^{}]*\}", body)
                assert block and block.group(0).count("pdl_launch_dependents") == 1, f.name
                assert body.count("pdl_launch_dependents") == 1, f.name
                checked += 1
    assert checked >= 4


class _EdgeData(ctypes.Structure):
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


def _overlapped_edges(call):
    """Number of programmatic edges in the graph that `call` captures to."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        keep = call()
    get_edges, handle, n = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2, ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert get_edges(handle, None, None, None, ctypes.byref(n)) == 0
    ends, data = [(ctypes.c_void_p * (n.value + 1))() for _ in range(2)], (_EdgeData * (n.value + 1))()
    assert get_edges(handle, ends[0], ends[1], data, ctypes.byref(n)) == 0
    del keep, graph
    return sum(d.type == 1 for d in data[:n.value])  # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(300, 512, 768), (300, 512, 32768), (300, 8192, 256)])
def test_no_overlap_beside_collectives(npu, capi, dev, shape):
    """The matmul launches of the all-reduce leave SMs to a collective: none may be placed early, whichever kernel takes the
    last, small chunk of rows (stream-K, tile, split-K); the same matmuls outside it are."""
    M, K, N = shape
    lib = capi.lib()
    uid = ctypes.create_string_buffer(capi.UNIQUE_ID_BYTES)
    capi.check(lib.qmm_comm_unique_id(uid), "qmm_comm_unique_id")
    capi.check(lib.qmm_comm_init_rank(b"overlap", uid, 1, 0), "qmm_comm_init_rank")
    try:
        a = torch.ones((M, K), dtype=torch.int8, device=dev)
        w = torch.ones((K, N), dtype=torch.int8, device=dev)
        scale, pt = torch.rand(N, device=dev), torch.rand(M, device=dev)
        assert _overlapped_edges(lambda: npu.npu_mm_all_reduce_base(a, w, "overlap", reduce_op="sum", dequant_scale=scale,
                                                                    pertoken_scale=pt, comm_turn=3)) == 0
        plain = lambda: [npu.npu_quant_matmul(a[:44], w, scale, pertoken_scale=pt[:44], output_dtype=torch.bfloat16)  # noqa: E731
                         for _ in range(2)]
        assert _overlapped_edges(plain) > 0
    finally:
        capi.check(lib.qmm_comm_destroy(b"overlap"), "qmm_comm_destroy")
