"""Outputs of the W8A8 kernels at the edges of their epilogue: rows that break TMA's 16-byte rules (odd widths with the
transposed weight view), partial tiles in both directions, every output type, scalar and per-column constants.  All
results are exact: integer sums, then fp32 operations with one rounding each in a fixed order."""
import ctypes
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float16, torch.int32, torch.int8])
@pytest.mark.parametrize("shape", [(1, 32, 17), (13, 256, 129), (31, 2064, 257), (128, 1040, 385), (129, 160, 255),
                                   (300, 144, 513), (300, 144, 512), (515, 272, 100), (40, 4096, 264)])
def test_edges(capi, oracle, dev, shape, out):
    M, K, N = shape
    g = torch.Generator().manual_seed(M * 31 + N)
    a = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8)
    wt = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8)  # stored [N, K], used as its transposed view
    pt = torch.rand(M, generator=g) * 1e-2 + 1e-3
    whole = not out.is_floating_point
    bias = torch.randint(-4096, 4096, (N,), generator=g, dtype=torch.int32) if whole else torch.randn(N, generator=g).to(out)
    for scalar in (False, True):
        n = 1 if scalar else N
        scale = torch.rand(n, generator=g) * (0.02 if out == torch.int8 else 1e-2) + 1e-4
        offset = torch.empty(n).uniform_(-9, 9, generator=g) if out == torch.int8 else None
        d = [t.to(dev) for t in (a, wt, scale, pt, bias)]
        if out == torch.int8:
            y = capi.quant_matmul_int8(d[0], d[1].t(), d[2], offset=offset.to(dev), pertoken_scale=d[3], bias=d[4])
        elif out == torch.int32:
            y = capi.quant_matmul(d[0], d[1].t(), None, bias=d[4], output_dtype=out)
        else:
            y = capi.quant_matmul(d[0], d[1].t(), d[2], pertoken_scale=d[3], bias=d[4], output_dtype=out)
        want = oracle.quant_matmul(a, wt.t(), scale, offset=offset, pertoken_scale=pt if out != torch.int32 else None,
                                   bias=bias, output_dtype=out)
        assert torch.equal(y.cpu(), want)


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float16, torch.int32, torch.int8])
@pytest.mark.parametrize("shape", [(1, 256, 512), (40, 4096, 272), (64, 1024, 1040), (128, 512, 128), (300, 256, 784)])
def test_output_pitch(capi, dev, shape, out):
    """Row-major weight, output rows at odd addresses (pitch N + 3, one element from the start of the buffer) through the C
    ABI: the bits of the contiguous call, and nothing written beside the rows."""
    M, K, N = shape
    g = torch.Generator(device=dev).manual_seed(M + N)
    a = torch.randint(-127, 128, (M, K), generator=g, device=dev, dtype=torch.int8)
    w = torch.randint(-127, 128, (K, N), generator=g, device=dev, dtype=torch.int8)
    scale, pt = torch.rand(N, generator=g, device=dev) * 1e-2, torch.rand(M, generator=g, device=dev) * 1e-2
    flat = torch.full((M * (N + 3) + 1,), 7, dtype=out, device=dev)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    at, stream, lib, n = ctypes.c_void_p(flat.data_ptr() + flat.element_size()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), capi.lib(), ctypes.c_size_t(0)
    if out == torch.int8:
        want = capi.quant_matmul_int8(a, w, scale, offset=scale, pertoken_scale=pt)
        capi.check(lib.qmm_quant_matmul_int8_workspace_size(M, N, K, ctypes.byref(n)), "size")
        ws = torch.zeros(n.value, dtype=torch.uint8, device=dev)
        capi.check(lib.qmm_quant_matmul_int8(ptr(a), K, ptr(w), N, 1, ptr(scale), N, ptr(scale), N, ptr(pt), None, at, N + 3, M, N, K,
                                             ptr(ws), n.value, stream), "matmul")
    else:
        whole = out == torch.int32
        want = capi.quant_matmul(a, w, None if whole else scale, pertoken_scale=None if whole else pt, output_dtype=out)
        capi.check(lib.qmm_quant_matmul_workspace_size(M, N, K, capi.ALGO_AUTO, ctypes.byref(n)), "size")
        ws = torch.zeros(max(n.value, 16), dtype=torch.uint8, device=dev)
        capi.check(lib.qmm_quant_matmul(ptr(a), K, ptr(w), N, 1, None if whole else ptr(scale), 0 if whole else N, None if whole else ptr(pt),
                                        None, capi.DTYPE_NONE, at, capi.dtype_code(out), N + 3, M, N, K, capi.ALGO_AUTO, ptr(ws), n.value,
                                        stream), "matmul")
    rows = flat[1:].view(M, N + 3)
    assert torch.equal(rows[:, :N], want)
    assert (rows[:, N:] == 7).all() and flat[0] == 7


def test_int8_stream_k_time(dev):
    """64 tokens, tiles shared by CTAs: the int8 output costs the stream-K kernel little more than the int32 one (1.28 times,
    with a clearing of its scratch; 1.62 when every element fetched the constants of its column again).  A small shape:
    the time of a large one depends on where its scratch lies."""
    sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "ascend-python_b200"))
    try:
        import torch_npu
    finally:
        sys.path.pop(0)
    M, K, N = 64, 1024, 1024
    g = torch.Generator(device=dev).manual_seed(3)
    a = torch.randint(-127, 128, (M, K), generator=g, device=dev, dtype=torch.int8)
    w = torch.randint(-127, 128, (N, K), generator=g, device=dev, dtype=torch.int8).t()
    scale, pt = torch.rand(N, device=dev) * 1e-2, torch.rand(M, device=dev) * 1e-2
    bias = torch.zeros(N, dtype=torch.int32, device=dev)

    def us(call):
        call()
        best = float("inf")
        for _ in range(7):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(4_000_000)
            s.record()
            for _ in range(20):
                call()
            e.record()
            torch.cuda.synchronize()
            best = min(best, s.elapsed_time(e) * 1e3 / 20)
        return best

    whole = us(lambda: torch_npu.npu_quant_matmul(a, w, scale, bias=bias, output_dtype=torch.int32))
    narrow = us(lambda: torch_npu.npu_quant_matmul(a, w, scale, offset=scale, pertoken_scale=pt, bias=bias, output_dtype=torch.int8))
    assert narrow < 1.45 * whole, f"int8 {narrow:.1f} us, int32 {whole:.1f} us"


@pytest.mark.parametrize("N", [16, 32, 48, 96, 112, 160, 208, 240, 272, 400, 496])
def test_tiles_that_end_inside_a_chunk(capi, dev, N):
    """Loads run one step ahead of their use: outputs whose last columns end in any 32 or 64 of a tile, in both kernels that share
    the epilogue, equal the dp4a kernel's (the same fp32 operations in the same order), bias and per-token scale included."""
    M, K = 300, 272
    g = torch.Generator(device=dev).manual_seed(N)
    a = torch.randint(-128, 128, (M, K), generator=g, device=dev, dtype=torch.int8)
    w = torch.randint(-128, 128, (K, N), generator=g, device=dev, dtype=torch.int8)
    scale, pt = torch.rand(N, generator=g, device=dev) * 1e-2, torch.rand(M, generator=g, device=dev)
    bias, ibias = torch.randn(N, generator=g, device=dev), torch.arange(N, device=dev, dtype=torch.int32) - 7
    for algo in (capi.ALGO_PAIR, capi.ALGO_TILE):
        for dtype, sc, p, b in ((torch.bfloat16, scale, pt, bias), (torch.float16, scale, None, bias.half()), (torch.int32, None, None, ibias)):
            got = capi.quant_matmul(a, w, sc, pertoken_scale=p, bias=b, output_dtype=dtype, algo=algo)
            assert torch.equal(got, capi.quant_matmul(a, w, sc, pertoken_scale=p, bias=b, output_dtype=dtype, algo=capi.ALGO_SIMT))
    assert capi.device_status() == 0


# More columns than the cluster kernel takes (148 x 256), so that the kernels which share the epilogue serve the call: stream-K
# (up to 16 rows), the one-CTA tile kernel (up to 128) and the CTA-pair kernel.  Ragged rows, one and several k blocks, columns that
# end 16, 112 and 128 into a tile, and (weight stored [N, K]) at odd ones, where output rows start at odd addresses.
@pytest.mark.parametrize("N,trans", [(37904, False), (38000, False), (38016, True), (37891, True)])
@pytest.mark.parametrize("M,K", [(1, 272), (16, 1040), (70, 272), (128, 128), (129, 272), (300, 400)])
def test_int8_output_of_the_kernels_beside_the_cluster_kernel(capi, dev, M, K, N, trans):
    """clamp(rint(float(acc + bias) * scale[n] * pertoken[m] + offset[n])), each operation rounded to fp32, over the exact sums of
    the dp4a kernel; with and without bias, offset and per-token scale."""
    g = torch.Generator(device=dev).manual_seed(M + K + N)
    a = torch.randint(-128, 128, (M, K), generator=g, device=dev, dtype=torch.int8)
    w = torch.randint(-128, 128, (N, K) if trans else (K, N), generator=g, device=dev, dtype=torch.int8)
    w = w.t() if trans else w
    acc = capi.quant_matmul(a, w, None, output_dtype=torch.int32, algo=capi.ALGO_SIMT)
    pt = torch.rand(M, generator=g, device=dev) + 0.5
    scale = (torch.rand(N, generator=g, device=dev) + 0.5) * (40.0 / (5400.0 * K ** 0.5))
    offset = torch.linspace(-30, 30, N, device=dev)
    bias = torch.randint(-4096, 4096, (N,), generator=g, device=dev, dtype=torch.int32)
    for p, o, b in ((pt, offset, bias), (None, None, None), (pt, None, bias), (None, offset, None)):
        want = (acc if b is None else acc + b).float() * scale
        want = want if p is None else want * p[:, None]
        want = want if o is None else want + o
        got = capi.quant_matmul_int8(a, w, scale, offset=o, pertoken_scale=p, bias=b)
        assert torch.equal(got, want.round().clamp(-128, 127).to(torch.int8))
    assert capi.device_status() == 0
