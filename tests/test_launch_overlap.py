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


class _Layer:
    """Two quantized projections and a W4A16 one behind norms, all of 1024 columns: every call reads what the call before
    wrote, and the allocator gives the buffers freed on the way out again."""

    def __init__(self, npu, dev, seed):
        g = torch.Generator(device=dev).manual_seed(seed)
        self.npu = npu
        self.w8 = torch.randint(-127, 128, (1024, 1024), generator=g, device=dev, dtype=torch.int8)
        self.scale = torch.rand(1024, generator=g, device=dev) * 1e-3 + 1e-4
        self.gamma = (torch.rand(1024, generator=g, device=dev) + 0.5).to(torch.bfloat16)
        self.w4 = torch.randint(-2 ** 31, 2 ** 31 - 1, (1024, 128), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
        self.s4 = (torch.rand((8, 1024), generator=g, device=dev) * 1e-2).to(torch.bfloat16)

    def steps(self, x, layers=3):
        """The calls one by one: yields after each, ends with the result."""
        npu = self.npu
        for _ in range(layers):
            q, s, _r = npu.npu_rms_norm_dynamic_quant(x, self.gamma)
            yield
            y = npu.npu_quant_matmul(q, self.w8, self.scale, pertoken_scale=s, output_dtype=torch.bfloat16)
            yield
            del q, s
            y, _r = npu.npu_rms_norm(y, self.gamma)
            yield
            q, s = npu.npu_dynamic_quant(y)
            yield
            y = npu.npu_quant_matmul(q, self.w8.t(), self.scale, pertoken_scale=s, output_dtype=torch.bfloat16)
            yield
            del q, s
            x = npu.npu_weight_quant_batchmatmul(y, self.w4, self.s4, antiquant_group_size=128)
            yield
        self.out = x

    def run(self, x, sync=False):
        for _ in self.steps(x):
            if sync:
                torch.cuda.synchronize()
        return self.out


ROWS = [1, 2, 5, 16, 64, 100, 300]  # every kernel of the two matmuls


@pytest.mark.gpu
@pytest.mark.parametrize("M", ROWS)
def test_chain_over_reused_buffers(npu, dev, M):
    """Calls that overlap give what calls one after the other give, also when the input is overwritten right behind them."""
    layer = _Layer(npu, dev, M)
    g = torch.Generator(device=dev).manual_seed(M)
    inputs = [torch.randn((M, 1024), generator=g, device=dev).to(torch.bfloat16) for _ in range(6)]
    want = [layer.run(x, sync=True).clone() for x in inputs]
    x = torch.empty_like(inputs[0])
    for _ in range(3):
        got = []
        for i in inputs:
            x.copy_(i)
            got.append(layer.run(x))
        assert all(torch.equal(a, b) for a, b in zip(want, got))


@pytest.mark.gpu
@pytest.mark.parametrize("M", ROWS)
def test_chain_captured(npu, dev, M):
    layer = _Layer(npu, dev, M + 100)
    x = torch.zeros((M, 1024), device=dev, dtype=torch.bfloat16)
    layer.run(x)  # weights prepacked
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = layer.run(x)
    g = torch.Generator(device=dev).manual_seed(M)
    for _ in range(4):
        value = torch.randn((M, 1024), generator=g, device=dev).to(torch.bfloat16)
        want = layer.run(value, sync=True).clone()
        x.copy_(value)
        graph.replay()
        got = y.clone()
        x.zero_()
        graph.replay()
        assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 16, 300])
def test_two_streams(npu, dev, M):
    layers = [_Layer(npu, dev, 7), _Layer(npu, dev, 8)]
    xs = [torch.randn((M, 1024), device=dev).to(torch.bfloat16) for _ in layers]
    want = [layer.run(x, sync=True).clone() for layer, x in zip(layers, xs)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(4):
        gens = [layer.steps(x) for layer, x in zip(layers, xs)]
        live = [True, True]
        while any(live):  # call by call in turn
            for i, gen in enumerate(gens):
                if live[i]:
                    with torch.cuda.stream(streams[i]):
                        live[i] = next(gen, "end") is None
        torch.cuda.synchronize()
        assert all(torch.equal(layer.out, w) for layer, w in zip(layers, want))


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 2])
def test_weight_rewritten_and_used_at_once(npu, dev, M):
    """One or two tokens read weights before they wait for the kernel in front (which has waited): a weight written again,
    and with it packed again, right before the call is the one that is used."""
    K = N = 2048
    g = torch.Generator(device=dev).manual_seed(5)
    x = torch.randn((M, K), generator=g, device=dev).to(torch.bfloat16)
    scale = (torch.rand((K // 128, N), generator=g, device=dev) * 1e-2).to(torch.bfloat16)
    ws = [torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
          for _ in range(4)]
    want = []
    for w in ws:
        torch.cuda.synchronize()
        want.append(npu.npu_weight_quant_batchmatmul(x, w, scale, antiquant_group_size=128))
    torch.cuda.synchronize()
    w = torch.zeros_like(ws[0])
    for _ in range(3):
        got = []
        for v in ws:
            w.copy_(v)
            got.append(npu.npu_weight_quant_batchmatmul(x, w, scale, antiquant_group_size=128))
        assert all(torch.equal(a, b) for a, b in zip(want, got))
