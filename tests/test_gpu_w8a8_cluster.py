"""The W8A8 kernel that cuts K over the CTA pairs of a cluster: sums exact, outputs equal to the dp4a kernel's (the same fp32
operations in the same order) at the edges of its tiles, slices and dispatch."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(dev, M, K, N, seed, trans):
    g = torch.Generator(device=dev).manual_seed(seed)
    a = torch.randint(-128, 128, (M, K), generator=g, device=dev, dtype=torch.int8)
    w = torch.randint(-128, 128, (N, K) if trans else (K, N), generator=g, device=dev, dtype=torch.int8)
    scale = torch.rand(N, generator=g, device=dev) * 1e-2 + 1e-3
    pt = torch.rand(M, generator=g, device=dev) * 0.1
    return a, w.t() if trans else w, scale, pt, torch.randn(N, generator=g, device=dev)


# token tiles of 32 .. 256 and their remainders, one k block to several a slice, ragged K and N, one slice to four; one wave with
# one cluster an SM pair and with two; whole tiles of padding columns (N = 16: the second CTA of a pair has none)
SHAPES = [(1, 16, 16), (1, 128, 240), (31, 144, 256), (32, 400, 272), (33, 4112, 528), (64, 8192, 256), (127, 1040, 1504),
          (128, 1024, 1024), (129, 2064, 784), (255, 4096, 1008), (256, 528, 2064), (257, 3072, 400), (333, 1024, 6144),
          (700, 2048, 1040), (1000, 512, 4096), (2048, 384, 1024), (1, 256, 148 * 256), (160, 272, 20000)]


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_against_dp4a_kernel(capi, dev, shape, trans):
    M, K, N = shape
    a, w, scale, pt, bias = _inputs(dev, M, K, N, M + K + N, trans)
    for algo in (capi.ALGO_CLUSTER, capi.ALGO_AUTO):
        ib = torch.arange(N, device=dev, dtype=torch.int32) - 7
        for b in (None, ib):
            got = capi.quant_matmul(a, w, None, bias=b, output_dtype=torch.int32, algo=algo)
            assert torch.equal(got, capi.quant_matmul(a, w, None, bias=b, output_dtype=torch.int32, algo=capi.ALGO_SIMT))
        for dtype, p, b in ((torch.bfloat16, pt, bias.bfloat16()), (torch.float16, None, bias), (torch.float16, pt, None)):
            got = capi.quant_matmul(a, w, scale, pertoken_scale=p, bias=b, output_dtype=dtype, algo=algo)
            want = capi.quant_matmul(a, w, scale, pertoken_scale=p, bias=b, output_dtype=dtype, algo=capi.ALGO_SIMT)
            assert torch.equal(got, want)
    assert capi.device_status() == 0


@pytest.mark.parametrize("shape", [(1, 16, 17), (33, 400, 257), (300, 1040, 1001), (128, 4096, 255)])
def test_odd_columns_int8_and_pitched_rows(capi, oracle, dev, shape):
    """Any number of columns (weight stored [N, K]); int8 outputs; outputs whose rows start at odd addresses."""
    M, K, N = shape
    a, w, scale, pt, bias = _inputs(dev, M, K, N, 3 * M + N, True)
    want = oracle.quant_matmul(a.cpu(), w.cpu(), scale.cpu(), pertoken_scale=pt.cpu(), bias=bias.cpu(), output_dtype=torch.bfloat16)
    got = capi.quant_matmul(a, w, scale, pertoken_scale=pt, bias=bias, output_dtype=torch.bfloat16, algo=capi.ALGO_CLUSTER)
    assert oracle.bf16_ulp_distance(got.cpu(), want).max().item() <= 1
    s8 = scale * (60.0 / (0.006 * 5400.0 * K ** 0.5)) / 0.05
    off = torch.linspace(-20, 20, N, device=dev)
    want8 = oracle.quant_matmul(a.cpu(), w.cpu(), s8.cpu(), pertoken_scale=pt.cpu(), offset=off.cpu(), output_dtype=torch.int8)
    assert torch.equal(capi.quant_matmul_int8(a, w, s8, offset=off, pertoken_scale=pt).cpu(), want8)
    for pitch, start in ((N + 3, 1), (N + 4, 2)):
        wide = torch.full((M * pitch + 8,), 7.0, device=dev, dtype=torch.bfloat16)
        rows = wide[start:start + M * pitch].view(M, pitch)
        capi.check(capi.lib().qmm_quant_matmul(
            capi._ptr(a), K, capi._ptr(w), 1, K, capi._ptr(scale), N, capi._ptr(pt), capi._ptr(bias), capi.DTYPE_F32,
            ctypes.c_void_p(rows.data_ptr()), capi.DTYPE_BF16, pitch, M, N, K, capi.ALGO_CLUSTER, None, 0, capi._stream()), "matmul")
        assert torch.equal(rows[:, :N], got)
        assert torch.all(rows[:, N:] == 7.0) and torch.all(wide[:start] == 7.0) and torch.all(wide[start + M * pitch:] == 7.0)


def test_shapes_beyond_one_wave_are_refused(capi, dev):
    """More tiles than clusters that are resident at once: an error by name, and another kernel by QMM_ALGO_AUTO."""
    a, w, scale, pt, bias = _inputs(dev, 64, 128, 148 * 256 + 16, 5, False)
    with pytest.raises(RuntimeError, match="cluster kernel"):
        capi.quant_matmul(a, w, None, output_dtype=torch.int32, algo=capi.ALGO_CLUSTER)
    got = capi.quant_matmul(a, w, None, output_dtype=torch.int32)
    assert torch.equal(got, capi.quant_matmul(a, w, None, output_dtype=torch.int32, algo=capi.ALGO_SIMT))


# What the plan makes of these on 148 SMs, token height / slices: 64 / 4, 64 / 2, 96 / 4 (three groups of tokens an owner), 96 / 2, 128 / 4,
# 128 / 2, 160 / 4, 160 / 2, 192 / 4, 192 / 2, 224 / 4, 256 / 2, and 256 / 4, whose received sums fill the operand ring
SLICED = [(250, 6144, 272), (100, 4096, 2064), (500, 8192, 272), (250, 4096, 2064), (100, 8192, 2064), (300, 6144, 2064),
          (130, 12288, 2000), (300, 6144, 4096), (500, 8192, 1040), (500, 8192, 2064), (200, 12288, 2064), (500, 12288, 4096),
          (250, 28672, 2064)]


@pytest.mark.parametrize("shape", SLICED)
def test_high_tiles_of_several_slices(capi, dev, shape):
    """The exchange of sums with several groups of tokens an owner, all four output types."""
    M, K, N = shape
    a, w, scale, pt, bias = _inputs(dev, M, K, N, M + K + N, M % 20 == 0)
    acc = capi.quant_matmul(a, w, None, output_dtype=torch.int32, algo=capi.ALGO_SIMT)
    assert torch.equal(capi.quant_matmul(a, w, None, output_dtype=torch.int32, algo=capi.ALGO_CLUSTER), acc)
    for dtype, p, b in ((torch.bfloat16, pt, bias.bfloat16()), (torch.float16, pt, None)):
        got = capi.quant_matmul(a, w, scale, pertoken_scale=p, bias=b, output_dtype=dtype, algo=capi.ALGO_CLUSTER)
        assert torch.equal(got, capi.quant_matmul(a, w, scale, pertoken_scale=p, bias=b, output_dtype=dtype, algo=capi.ALGO_SIMT))
    s8, off = scale * (8000.0 / (5400.0 * K ** 0.5)), torch.linspace(-20, 20, N, device=dev)
    ib = torch.arange(N, device=dev, dtype=torch.int32) - 7
    got = capi.quant_matmul_int8(a, w, s8, offset=off, pertoken_scale=pt * 10, bias=ib)
    want = (acc + ib).float() * s8 * (pt * 10)[:, None] + off
    assert torch.equal(got, want.round().clamp(-128, 127).to(torch.int8))
    assert capi.device_status() == 0


@pytest.mark.parametrize("shape", [(145, 20608, 19440), (300, 24576, 14064)])
def test_time_of_lower_tiles_over_a_long_k(capi, dev, shape):
    """Tiles of 160 tokens, two on some SMs and one on others, K of more than 160 blocks: the kernel that is chosen is the faster one of
    the cluster and CTA-pair kernels (0.65 to 0.72 of the other's time), with a tenth for noise."""
    M, K, N = shape
    a, w, scale, pt, _ = _inputs(dev, M, K, N, 1, True)

    def us(algo):
        best = float("inf")
        for _ in range(7):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            capi.quant_matmul(a, w, scale, pertoken_scale=pt, output_dtype=torch.bfloat16, algo=algo)
            s.record()
            for _ in range(5):
                capi.quant_matmul(a, w, scale, pertoken_scale=pt, output_dtype=torch.bfloat16, algo=algo)
            e.record()
            torch.cuda.synchronize()
            best = min(best, s.elapsed_time(e) * 1e3 / 5)
        return best

    chosen, cluster, pair = (us(algo) for algo in (capi.ALGO_AUTO, capi.ALGO_CLUSTER, capi.ALGO_PAIR))
    assert chosen < 1.1 * min(cluster, pair), f"chosen {chosen:.1f} us, cluster {cluster:.1f}, pair {pair:.1f}"
