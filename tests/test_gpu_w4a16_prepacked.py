"""Prepacked W4A16 path on the GPU: the layout pass round-trips bit-exactly, and the matmul over the
prepacked stream meets the same bound against the fp64 oracle as the stock entry point.

Tolerance (floating point, stated here).  The kernel rounds every weight W = fma(w, scale, offset*scale) once
to the activation dtype before the tensor-core product (a relative perturbation of at most u = 2^-9 for bf16,
2^-12 for f16), accumulates in fp32 and rounds the output once (u again).  The error of an output is therefore
a sum of K independent terms x[m,k] * dW[k,n]; its standard deviation is about 0.45 u * rss with
rss[m,n] = sqrt(sum_k (x[m,k] * W[k,n])^2), the natural scale of accumulated rounding error (a bound relative
to the row's rms would be too tight for columns whose scales are above average and too loose for the others).
The bound asserted is
    |y - y_ref| <= 2 u * |y_ref| + 8 u * rss[m,n]             (u = 2^-9 bf16, 2^-12 f16)
i.e. the output rounding plus about 18 standard deviations of the accumulated weight rounding.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rss(oracle, x, packed_w, scale, offset, group):
    W = oracle.antiquant_weight(packed_w, scale, offset, group)
    return np.sqrt((x.double().numpy() ** 2) @ (W ** 2))


def _assert_close(y, y_ref, rss, dtype):
    u = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    y = y.detach().float().cpu().numpy().astype(np.float64)
    bound = 2 * u * np.abs(y_ref) + 8 * u * rss + 1e-30
    worst = np.max(np.abs(y - y_ref) / bound)
    assert worst <= 1.0, f"error is {worst:.2f}x the bound"


@pytest.mark.parametrize("shape", [(128, 64, 128), (256, 136, 128), (1024, 4096, 256), (8192, 2048 + 32, 128),
                                   (384, 8, 384)])
def test_prepack_round_trip(capi, oracle, dev, shape):
    """unpack(prepack(w)) == w, and the scale / offset*scale rows of every block are what the layout says."""
    K, N, group = shape
    _, packed_w, scale, offset = oracle.make_w4a16_inputs(1, K, N, seed=K + N, group=group)
    buf = capi.w4a16_prepack(packed_w.to(dev), scale.to(dev), offset.to(dev), group_size=group)
    tiles, chunks = (N + 127) // 128, K // 128
    padded = 2 * ((chunks + 1) // 2)  # blocks along K come in pairs; an odd count is padded with a zero block
    assert buf.numel() == capi.w4a16_prepack_size(N, K, group) == tiles * padded * 8704
    back = capi.w4a16_unpack_weight(buf, N, K)
    assert torch.equal(back.cpu(), packed_w)
    blocks = buf.cpu().view(-1, 8704)
    so = blocks[:, 8192:].contiguous().view(torch.bfloat16).view(tiles, padded, 2, 128)
    s_ref = torch.zeros((padded, tiles * 128), dtype=torch.bfloat16)
    t_ref = torch.zeros_like(s_ref)
    rows = torch.arange(chunks) * 128 // group
    s_ref[:chunks, :N] = scale[rows]
    t_ref[:chunks, :N] = (offset[rows].float() * scale[rows].float()).to(torch.bfloat16)
    assert torch.equal(so[:, :, 0, :].permute(1, 0, 2).reshape(padded, -1), s_ref)
    assert torch.equal(so[:, :, 1, :].permute(1, 0, 2).reshape(padded, -1), t_ref)
    if padded > chunks:
        assert not blocks.view(tiles, padded, 8704)[:, chunks:].any()


def test_prepack_refusals(capi, dev):
    assert capi.w4a16_prepack_size(256, 192, 64) == 0      # K not a multiple of 128
    assert capi.w4a16_prepack_size(256, 256, 64) == 0      # group not a multiple of 128
    assert capi.w4a16_prepack_size(256, 512, 0) > 0        # per-channel: group = K
    w = torch.zeros((192, 32), dtype=torch.int32, device=dev)
    s = torch.ones((1, 256), dtype=torch.bfloat16, device=dev)
    with pytest.raises(capi.QmmError):
        capi.w4a16_prepack(w, s, None, group_size=0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 256, 64, 128), (2, 384, 200, 128), (2, 8192, 1024, 256), (4, 256, 128, 128), (16, 1024, 512, 128), (64, 2048, 1024, 128),
                                   (130, 512, 256, 128), (8, 512, 256, 512), (33, 4096, 7168, 128),
                                   (5, 8192, 2048 + 32, 128), (64, 1024, 4096, 1024), (12, 256, 8, 256),
                                   (16, 2048, 1024 + 72, 128), (48, 1152, 640, 384)])
def test_against_oracle(capi, oracle, dev, shape, dtype):
    M, K, N, group = shape
    x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=M + K + N, group=group, dtype=dtype)
    y_ref = oracle.weight_quant_batchmatmul(x, packed_w, scale, offset, antiquant_group_size=group)
    rss = _rss(oracle, x, packed_w, scale, offset, group)
    buf = capi.w4a16_prepack(packed_w.to(dev), scale.to(dev), offset.to(dev), group_size=group)
    for _ in range(2):  # the second call reuses the scratch the first one left
        y = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N)
        assert y.dtype == dtype and y.shape == (M, N)
        _assert_close(y, y_ref, rss, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 256, 64, 128), (2, 384, 200, 128), (2, 8192, 1024, 256), (1, 4096, 7168, 128),
                                   (2, 1024, 4096, 1024),
                                   # one block and its padding; slices of K: eight up to 30 tiles, four up to 66, two up to 148;
                                   # a long K whose digits leave a short ring; more tiles than SMs; beyond the tile kernel's range
                                   (1, 128, 8, 128), (2, 4096, 30 * 128, 128), (1, 4096, 30 * 128 + 8, 128),
                                   (2, 2176, 66 * 128, 128), (1, 2048, 66 * 128 + 16, 2048), (1, 1152, 148 * 128, 128),
                                   (2, 1024, 148 * 128 + 8, 128), (2, 65536, 136, 128), (2, 8192, 9280, 128),
                                   (1, 2176, 37 * 128 - 8, 128), (2, 4096, 18 * 128, 128)])  # clusters that need two CTAs an SM
def test_one_or_two_tokens_meet_the_stock_tolerance(capi, oracle, dev, shape, dtype):
    """One or two tokens take the integer dot-product kernel, which never rounds a weight: it meets the bound of
    the stock-layout kernels, |y - y_ref| <= 2 u |y_ref| + 2^-7 (u / 2^-9) rms(row), not only the rss bound."""
    M, K, N, group = shape
    x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=M + K + N, group=group, dtype=dtype)
    y_ref = oracle.weight_quant_batchmatmul(x, packed_w, scale, offset, antiquant_group_size=group)
    buf = capi.w4a16_prepack(packed_w.to(dev), scale.to(dev), offset.to(dev), group_size=group)
    y = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N).float().cpu().numpy()
    u = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    rms = np.sqrt(np.mean(y_ref ** 2, axis=1, keepdims=True))
    assert np.all(np.abs(y - y_ref) <= 2 * u * np.abs(y_ref) + 2.0 ** -7 * (u / 2.0 ** -9) * rms + 1e-30)


def test_bias_and_no_offset(capi, oracle, dev):
    x, packed_w, scale, _ = oracle.make_w4a16_inputs(5, 512, 256, seed=3)
    bias = torch.randn(256).to(torch.bfloat16)
    y_ref = oracle.weight_quant_batchmatmul(x, packed_w, scale, None, bias=bias, antiquant_group_size=128)
    buf = capi.w4a16_prepack(packed_w.to(dev), scale.to(dev), None, group_size=128)
    y = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, 256, bias=bias.to(dev))
    _assert_close(y, y_ref, _rss(oracle, x, packed_w, scale, None, 128), torch.bfloat16)


@pytest.mark.parametrize("M", [1, 2, 16, 64])
def test_decode_full_size(capi, oracle, dev, M):
    """K = 8192, N = 28672, group 128: oracle on a sample of 8-column groups, linearity over the whole output
    (f(2x) == 2 f(x) exactly: scaling by two commutes with every rounding), and run-to-run identity."""
    K, N, group = 8192, 28672, 128
    g = torch.Generator(device=dev).manual_seed(M)
    x = torch.randn((M, K), generator=g, device=dev, dtype=torch.float32).to(torch.bfloat16)
    packed_w = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    scale = torch.empty((K // group, N), device=dev).uniform_(5e-3, 2e-2, generator=g).to(torch.bfloat16)
    offset = torch.empty((K // group, N), device=dev).uniform_(-1, 1, generator=g).to(torch.bfloat16)
    buf = capi.w4a16_prepack(packed_w, scale, offset, group_size=group)
    assert torch.equal(capi.w4a16_unpack_weight(buf, N, K), packed_w)
    y = capi.weight_quant_batchmatmul_prepacked(x, buf, N)
    y_again = capi.weight_quant_batchmatmul_prepacked(x, buf, N)
    assert torch.equal(y, y_again)
    y2 = capi.weight_quant_batchmatmul_prepacked(x * 2, buf, N)
    assert torch.equal(y2.float(), y.float() * 2)
    words = torch.arange(1, N // 8, 97, device=dev)
    cols = (words[:, None] * 8 + torch.arange(8, device=dev)[None, :]).reshape(-1)
    y_ref = oracle.weight_quant_batchmatmul(x.cpu(), packed_w[:, words].cpu(), scale[:, cols].cpu(),
                                            offset[:, cols].cpu(), antiquant_group_size=group)
    rss = _rss(oracle, x.cpu(), packed_w[:, words].cpu(), scale[:, cols].cpu(), offset[:, cols].cpu(), group)
    _assert_close(y[:, cols], y_ref, rss, torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(65, 128, 136, 128), (128, 640, 8, 640), (129, 1152, 264, 384), (255, 384, 1032, 128),
                                   (257, 256, 19200, 256), (600, 512, 1152, 512), (1030, 128, 136, 128)])
def test_more_than_64_rows(capi, oracle, dev, shape, dtype):
    """The wide form: one to five row tiles, ragged last ones, odd numbers of blocks, fewer output tiles than SMs and more,
    on 148 SMs all of them whole tiles; and a result that two calls repeat."""
    M, K, N, group = shape
    x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=M + K + N, group=group, dtype=dtype)
    y_ref = oracle.weight_quant_batchmatmul(x, packed_w, scale, offset, antiquant_group_size=group)
    buf = capi.w4a16_prepack(packed_w.to(dev), scale.to(dev), offset.to(dev), group_size=group)
    y = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N)
    _assert_close(y, y_ref, _rss(oracle, x, packed_w, scale, offset, group), dtype)
    assert torch.equal(y, capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N))


@pytest.mark.parametrize("shape", [(3, 8192, 1024), (16, 8192, 1024), (64, 2304, 7168), (33, 28672, 1024)])
def test_cut_points_up_to_64_rows(capi, dev, shape):
    """Where the K sum of a tile is cut into partial sums decides its last bits: CTA c of G takes the block pairs
    [total * c / G, total * (c + 1) / G).  One nonzero k per block pair (256 k), values 2^25, 2, 2, ..., 2, -2^25: a 2 is
    lost in a sum that holds 2^25 (half of its unit, to even or cut off) and kept in one that starts after a cut, so the
    output counts the pairs behind the cuts.  The sums below are exact or round as said; the output is a small integer."""
    M, K, N = shape
    pairs, tiles = K // 256, N // 128
    total = pairs * tiles
    G = min(total, torch.cuda.get_device_properties(dev).multi_processor_count)
    assert total % G != 0
    v = np.full(pairs, 2.0, dtype=np.float32)
    v[0], v[-1] = 2.0 ** 25, -2.0 ** 25
    x = torch.zeros((M, K), dtype=torch.bfloat16)
    x[:, 5::256] = torch.from_numpy(v).to(torch.bfloat16)
    w = torch.full((K, N // 8), 0x11111111, dtype=torch.int32)
    buf = capi.w4a16_prepack(w.to(dev), torch.ones((1, N), dtype=torch.bfloat16, device=dev), None, group_size=0)
    y = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N).float().cpu().numpy()
    cuts = sorted({total * c // G for c in range(G + 1)} | {t * pairs for t in range(tiles + 1)})
    expect = np.zeros(tiles, dtype=np.float32)
    for a, b in zip(cuts, cuts[1:]):
        part = np.float32(0)
        for i in range(a, b):
            part = np.float32(part + v[i % pairs])
        expect[a // pairs] = np.float32(expect[a // pairs] + part)
    assert len(np.unique(expect)) > 1
    np.testing.assert_array_equal(y, np.broadcast_to(np.repeat(expect, 128), (M, N)))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(65, 8192, 136, 128), (200, 4096, 264, 4096), (257, 28672, 1032, 128),
                                   (520, 2560, 12808, 256), (600, 4096, 1152, 128)])
def test_more_than_64_rows_shared_tiles(capi, oracle, dev, shape, dtype):
    """The wide form with equal shares: many CTAs a tile, several row tiles with a ragged last one, and tiles of two CTAs
    whose ranges end inside them (on 148 SMs).  Bias; the second call finds the first one's counters; a call with another
    plan (whole tiles) on the same scratch in between."""
    M, K, N, group = shape
    x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=M + K + N, group=group, dtype=dtype)
    bias = torch.randn(N, generator=torch.Generator().manual_seed(N)).to(dtype)
    buf = capi.w4a16_prepack(packed_w.to(dev), scale.to(dev), offset.to(dev), group_size=group)
    xd, bd = x.to(dev), bias.to(dev)
    y = capi.weight_quant_batchmatmul_prepacked(xd, buf, N, bias=bd)
    # a sample of columns: every tile's edges and something between
    cols = sorted({c for c in range(0, N, 128)} | {min(c + 127, N - 1) for c in range(0, N, 128)} | set(range(64, N, 509)))
    words = sorted({c // 8 for c in cols})
    cols = torch.tensor([8 * i + j for i in words for j in range(8)])
    y_ref = oracle.weight_quant_batchmatmul(x, packed_w[:, words], scale[:, cols], offset[:, cols], bias=bias[cols],
                                            antiquant_group_size=group)
    rss = _rss(oracle, x, packed_w[:, words], scale[:, cols], offset[:, cols], group)
    _assert_close(y[:, cols.to(dev)], y_ref, rss, dtype)
    capi.weight_quant_batchmatmul_prepacked(torch.ones((65, 256), dtype=dtype, device=dev),
                                            torch.zeros(capi.w4a16_prepack_size(19200, 256, 256), dtype=torch.uint8, device=dev), 19200)
    assert torch.equal(y, capi.weight_quant_batchmatmul_prepacked(xd, buf, N, bias=bd))


@pytest.mark.parametrize("shape", [(65, 256, 136), (96, 2048, 19208), (200, 4096, 264), (600, 4096, 1152), (33, 1024, 264)])
def test_row_pitches_and_unaligned_output(capi, dev, shape):
    """Rows of x with a pitch, rows of the output at odd addresses (stores element by element), with bias, through the C ABI:
    the bits of the contiguous call, and nothing written beside the rows.  Whole and shared tiles."""
    M, K, N = shape
    g = torch.Generator(device=dev).manual_seed(M)
    x = torch.randn((M, K), generator=g, device=dev).to(torch.bfloat16)
    w = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    scale = (torch.rand((K // 128, N), generator=g, device=dev) * 1e-2).to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device=dev).to(torch.bfloat16)
    buf = capi.w4a16_prepack(w, scale, None, group_size=128)
    want = capi.weight_quant_batchmatmul_prepacked(x, buf, N, bias=bias)
    xp = torch.full((M, K + 24), float("nan"), dtype=torch.bfloat16, device=dev)
    xp[:, :K] = x
    flat = torch.full((M * (N + 5) + 1,), 7.0, dtype=torch.bfloat16, device=dev)
    n = ctypes.c_size_t(0)
    capi.check(capi.lib().qmm_weight_quant_batchmatmul_prepacked_workspace_size(M, N, K, ctypes.byref(n)), "size")
    ws = torch.zeros(n.value, dtype=torch.uint8, device=dev)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    for _ in range(2):
        capi.check(capi.lib().qmm_weight_quant_batchmatmul_prepacked(
            ptr(xp), capi.dtype_code(torch.bfloat16), K + 24, ptr(buf), buf.numel(), ptr(bias),
            ctypes.c_void_p(flat.data_ptr() + 2), N + 5, M, N, K, ptr(ws), n.value,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "matmul")
        rows = flat[1:].view(M, N + 5)
        assert torch.equal(rows[:, :N], want)
        assert (rows[:, N:] == 7.0).all() and flat[0] == 7.0


def test_slots_of_the_ring_belong_to_one_group(capi, oracle, dev):
    """Rings of three to fifteen blocks, many calls back to back: every call the same bits, no wait that ran out."""
    for M, K, N in ((2, 28672, 2048), (1, 384, 4096), (2, 8192, 4096), (1, 14336, 1024), (2, 57344, 256)):
        x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=K, group=128)
        buf = capi.w4a16_prepack(packed_w.to(dev), scale.to(dev), offset.to(dev), group_size=128)
        xd = x.to(dev)
        first = capi.weight_quant_batchmatmul_prepacked(xd, buf, N)
        for _ in range(200):
            last = capi.weight_quant_batchmatmul_prepacked(xd, buf, N)
        assert torch.equal(first, last)
    assert capi.device_status() == 0


@pytest.mark.parametrize("N", [8, 120, 128, 520, 1032])
def test_prepack_of_a_pitched_or_unaligned_weight(capi, oracle, dev, N):
    """Rows of the packed weight that do not start on 16 bytes, or have columns of another tensor behind them, pack the same."""
    K = 384
    _, packed_w, scale, offset = oracle.make_w4a16_inputs(1, K, N, seed=N, group=128)
    w, sc, of = packed_w.to(dev), scale.to(dev), offset.to(dev)
    want = capi.w4a16_prepack(w, sc, of, group_size=128)
    assert torch.equal(capi.w4a16_unpack_weight(want, N, K).cpu(), packed_w)
    for pitch, start in ((N // 8 + 3, 1), (N // 8 + 4, 0), (N // 8 + 4 - N // 8 % 4, 4)):
        flat = torch.full((K * pitch + 8,), -1, dtype=torch.int32, device=dev)
        rows = flat[start:start + K * pitch].view(K, pitch)[:, :N // 8]
        rows.copy_(w)
        got = torch.empty_like(want)
        capi.check(capi.lib().qmm_w4a16_prepack(ctypes.c_void_p(rows.data_ptr()), pitch, capi._ptr(sc), capi._ptr(of), capi.DTYPE_BF16,
                                                128, N, K, capi._ptr(got), got.numel(), capi._stream()), "prepack")
        assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(3, 128, 8, 128), (8, 384, 200, 128), (5, 1152, 4104, 384), (4, 8192, 1024, 256), (7, 2048, 136, 2048),
                                   (16, 1024, 1032, 128), (9, 640, 20008, 128)])
def test_few_tokens_with_tables_meet_the_stock_tolerance(capi, oracle, dev, shape, dtype):
    """Three to sixteen rows with the tables at hand: the weight is never rounded, so the stock layout's bound holds (see above);
    with and without offset and bias; tables at odd addresses are not used, which leaves the bound of the rounded weight."""
    M, K, N, group = shape
    x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=M + K + N, group=group, dtype=dtype)
    bias = torch.randn(N, generator=torch.Generator().manual_seed(N)).to(dtype)
    u = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    for off, b in ((offset, None), (None, bias)):
        y_ref = oracle.weight_quant_batchmatmul(x, packed_w, scale, off, bias=b, antiquant_group_size=group)
        sd, od = scale.to(dev), None if off is None else off.to(dev)
        buf = capi.w4a16_prepack(packed_w.to(dev), sd, od, group_size=group)
        got = [capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N, bias=None if b is None else b.to(dev), tables=(sd, od, group))
               for _ in range(20)]
        assert all(torch.equal(got[0], g) for g in got)
        y = got[0].float().cpu().numpy()
        rms = np.sqrt(np.mean(y_ref ** 2, axis=1, keepdims=True))
        assert np.all(np.abs(y - y_ref) <= 2 * u * np.abs(y_ref) + 2.0 ** -7 * (u / 2.0 ** -9) * rms + 1e-30)
        shifted = torch.empty(sd.numel() + 1, dtype=dtype, device=dev)
        shifted[1:] = sd.flatten()
        y1 = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N, bias=None if b is None else b.to(dev), tables=(shifted[1:], od, group))
        _assert_close(y1, y_ref, _rss(oracle, x, packed_w, scale, off, group), dtype)
    assert capi.device_status() == 0


@pytest.mark.parametrize("shape", [(4, 256, 136), (6, 4096, 1032), (8, 640, 2056)])
def test_few_tokens_infinities_and_nans(capi, oracle, dev, shape):
    """An infinity in a row makes its outputs infinite with the weight's sign, two of them or a NaN what plain arithmetic makes
    of it, and leaves the other rows alone: whole tiles and tiles that CTAs share."""
    M, K, N = shape
    x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=K, group=128)
    clean = x.clone()
    x[0, 3], x[1, K - 1] = float("inf"), float("-inf")
    x[2, 5], x[2, 9] = float("inf"), float("-inf")
    x[3, 7] = float("nan")
    sd, od = scale.to(dev), offset.to(dev)
    buf = capi.w4a16_prepack(packed_w.to(dev), sd, od, group_size=128)
    W = torch.from_numpy(np.asarray(oracle.antiquant_weight(packed_w, scale, offset, 128), dtype=np.float32))
    want = (x.float()[:4, :, None] * W[None]).sum(dim=1)
    y = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N, tables=(sd, od, 128)).float().cpu()
    assert torch.equal(torch.isnan(y[:4]), torch.isnan(want)) and torch.equal(torch.isinf(y[:4]), torch.isinf(want))
    assert torch.equal(torch.sign(y[:2]), torch.sign(want[:2]))
    y_clean = capi.weight_quant_batchmatmul_prepacked(clean.to(dev), buf, N, tables=(sd, od, 128)).float().cpu()
    assert torch.equal(y[4:], y_clean[4:])


def test_operator_takes_few_rows_of_any_width(oracle, dev):
    """npu_weight_quant_batchmatmul with 3 to 8 rows: widths whose packed rows TMA cannot address, small and large, x at an odd
    address; never further from 64 bits than the stock layout's bound."""
    import sys
    from pathlib import Path

    sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "ascend-python_b200"))
    try:
        import torch_npu
    finally:
        sys.path.pop(0)
    for M, K, N, group in ((3, 1024, 1024, 128), (8, 4096, 6144, 128), (5, 4096, 6176, 128), (3, 384, 1000, 0), (8, 2048, 13528, 128), (4, 192, 72, 64)):
        x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=M + N, group=group or K)
        y_ref = oracle.weight_quant_batchmatmul(x, packed_w, scale, offset, antiquant_group_size=group or K)
        rms = np.sqrt(np.mean(y_ref ** 2, axis=1, keepdims=True))
        flat = torch.empty(M * K + 1, dtype=x.dtype, device=dev)
        flat[1:] = x.to(dev).flatten()
        for xd in (x.to(dev), flat[1:].view(M, K)):
            y = torch_npu.npu_weight_quant_batchmatmul(xd, packed_w.to(dev), scale.to(dev), offset.to(dev), antiquant_group_size=group)
            assert np.all(np.abs(y.float().cpu().numpy() - y_ref) <= 2.0 ** -8 * np.abs(y_ref) + 2.0 ** -7 * rms)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(3, 512, 136), (8, 4096, 1032)])
def test_few_tokens_one_large_activation_a_block(capi, oracle, dev, shape, dtype):
    """Every 128th activation is 16384 and meets weights of zero, the others are near 1/64: the sum of the others is left as it is.
    Bound: the output's rounding, and K roundings of fp32 sums of what is summed (a zero times 16384 counts as 1 at most, the
    smallest exponent of an f16)."""
    M, K, N = shape
    x, packed_w, scale, _ = oracle.make_w4a16_inputs(M, K, N, seed=K + N, group=128, dtype=dtype)
    x = (x.float() / 64).to(dtype)
    x[:, ::128] = 16384
    packed_w[::128] = 0
    y_ref = oracle.weight_quant_batchmatmul(x, packed_w, scale, None, antiquant_group_size=128)
    sums = np.abs(x.double().numpy()) @ np.abs(np.asarray(oracle.antiquant_weight(packed_w, scale, None, 128), dtype=np.float64))
    sd = scale.to(dev)
    buf = capi.w4a16_prepack(packed_w.to(dev), sd, None, group_size=128)
    y = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N, tables=(sd, None, 128)).float().cpu().numpy()
    u = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    bound = 2 * u * np.abs(y_ref) + K * 2.0 ** -23 * (sums + scale.float().max().item())
    assert np.all(np.abs(y - y_ref) <= bound), f"error is {np.max(np.abs(y - y_ref) / bound):.1f}x the bound"


@pytest.mark.parametrize("shape", [(4, 256, 136), (6, 4096, 1032)])
def test_few_tokens_sums_beyond_fp32(capi, oracle, dev, shape):
    """Activations of up to 2^124 in one row: sums of products with whole-number weights leave the range of fp32, the outputs (the
    scales are near 2^-7) do not.  Bound: the output's rounding and K roundings of the fp32 sums.  The other rows stay as they are."""
    M, K, N = shape
    x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=K + 1, group=128)
    clean = x.clone()
    x[1] = (x[1].float().clamp(-4, 4) * 2.0 ** 122).to(torch.bfloat16)
    y_ref = oracle.weight_quant_batchmatmul(x, packed_w, scale, offset, antiquant_group_size=128)
    assert np.abs(y_ref).max() < 2.0 ** 127
    sums = np.abs(x.double().numpy()) @ np.abs(np.asarray(oracle.antiquant_weight(packed_w, scale, offset, 128), dtype=np.float64))
    sd, od = scale.to(dev), offset.to(dev)
    buf = capi.w4a16_prepack(packed_w.to(dev), sd, od, group_size=128)
    y = capi.weight_quant_batchmatmul_prepacked(x.to(dev), buf, N, tables=(sd, od, 128)).cpu()
    y_clean = capi.weight_quant_batchmatmul_prepacked(clean.to(dev), buf, N, tables=(sd, od, 128)).cpu()
    others = [m for m in range(M) if m != 1]
    assert torch.equal(y[others], y_clean[others])
    error = np.abs(y[1].double().numpy() - y_ref[1])
    assert np.all(error <= 2.0 ** -8 * np.abs(y_ref[1]) + K * 2.0 ** -23 * sums[1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(8, 512, 136), (8, 4096, 4096), (7, 256, 40008)])  # the last: several tiles a CTA
def test_few_tokens_not_finite_rows_and_bias(capi, oracle, dev, shape, dtype):
    """Rows with activations or columns with a bias that is not finite: infinities, their signs and NaN as plain arithmetic has them,
    everything else as without them, and in little more than the time of finite ones (twice, and 10 us)."""
    M, K, N = shape
    x, packed_w, scale, offset = oracle.make_w4a16_inputs(M, K, N, seed=K + N, group=128, dtype=dtype)
    w = torch.from_numpy(np.asarray(oracle.antiquant_weight(packed_w, scale, offset, 128), dtype=np.float64))
    sd, od = scale.to(dev), offset.to(dev)
    buf = capi.w4a16_prepack(packed_w.to(dev), sd, od, group_size=128)

    def call(xd, b):
        return capi.weight_quant_batchmatmul_prepacked(xd, buf, N, bias=b, tables=(sd, od, 128))

    def us(xd, b):
        call(xd, b)
        best = float("inf")
        for _ in range(7):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(4_000_000)
            s.record()
            for _ in range(20):
                call(xd, b)
            e.record()
            torch.cuda.synchronize()
            best = min(best, s.elapsed_time(e) * 1e3 / 20)
        return best

    bias = torch.zeros(N, dtype=dtype)
    bias[::2] = float("-inf")
    bad = x.clone()
    bad[0, K // 2 + 5] = float("nan")
    bad[1, ::131] = float("inf")
    bad[2, K - 1] = float("-inf")
    bad[4, 0], bad[4, K - 1] = float("inf"), float("nan")
    bad[6, :] = float("nan")
    clean = call(x.to(dev), None)
    for xs, b in ((bad, None), (x, bias), (bad, bias)):
        xd, bd = xs.to(dev), None if b is None else b.to(dev)
        y = call(xd, bd).cpu()
        want = xs.double() @ w + (0 if b is None else b.double())
        special = ~torch.isfinite(want)
        assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isfinite(y), ~special)
        assert torch.equal(torch.sign(y[torch.isinf(want)]).double(), torch.sign(want[torch.isinf(want)]))
        assert torch.equal(y[~special], clean.cpu()[~special])
        assert us(xd, bd) < 2 * us(x.to(dev), None if b is None else torch.zeros_like(bd)) + 10


def test_few_tokens_not_finite_many_tiles_a_cta(capi, dev):
    """More tiles a CTA than it notes one by one (33 of whole K): as calls over 148 tiles each, a tile a CTA, have it."""
    M, K, part = 4, 256, 148 * 128
    N = 33 * part - 40
    g = torch.Generator(device=dev).manual_seed(9)
    w = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    scale = (torch.rand((K // 128, N), generator=g, device=dev) * 1e-2 + 1e-3).bfloat16()
    x = torch.randn((M, K), generator=g, device=dev).bfloat16()
    x[0, 5], x[1, 200], x[1, 3] = float("inf"), float("inf"), float("-inf")
    x[2] = (x[2].float().clamp(-4, 4) * 2.0 ** 122).bfloat16()

    def call(lo, hi):
        s = scale[:, lo:hi].contiguous()
        buf = capi.w4a16_prepack(w[:, lo // 8:hi // 8].contiguous(), s, None, group_size=128)
        return capi.weight_quant_batchmatmul_prepacked(x, buf, hi - lo, tables=(s, None, 128))

    whole, again = call(0, N), call(0, N)
    parts = torch.cat([call(lo, min(lo + part, N)) for lo in range(0, N, part)], dim=1)
    for y in (whole, again):
        assert torch.equal(torch.isnan(y), torch.isnan(parts))
        assert torch.equal(torch.nan_to_num(y), torch.nan_to_num(parts))
    assert torch.isfinite(parts[2:]).all()
