// Fused dequantization epilogue shared by every W8A8 kernel.
//
//   out_dtype int32 : out = acc (+ int32 bias)
//   bf16, f16       : out = cast(float(acc) * scale[n] * pertoken_scale[m] + float(bias[n]))
//   int8            : out = clamp(rint(float(acc + int32 bias) * scale[n] * pertoken_scale[m] + offset[n]), -128, 127)
// evaluated in fp32 with one rounding per operation in exactly this order, so
// that the result equals the CPU oracle's fp32 epilogue bit for bit before the
// final round-to-nearest-even conversion to bf16/f16.
#pragma once

#include "qmm_common.cuh"

namespace qmm {

struct EpilogueParams {
    const float *scale;           // [N] or [1]
    const float *pertoken_scale;  // [M] or nullptr
    const void *bias;             // [N] or nullptr
    int bias_dtype;               // QMM_DTYPE_* or QMM_DTYPE_NONE
    int scale_is_scalar;          // scale has a single element
    void *out;
    int64_t ld_out;
    int64_t M;
    int64_t N;
    const float *offset = nullptr;  // [N] or [1] or nullptr; int8 output only
    int offset_is_scalar = 0;
};

// out_dtype of quant_matmul_dispatch for the int8 output (the C ABI has an entry point of its own for it)
constexpr int kOutI8 = 100;

// Row-parallel matmul whose output tiles go straight to the rank that will reduce them: rank o owns the
// rows [o * rows_per, (o+1) * rows_per) and receives them from rank s at
// base[o] + area_off + s * rows_per * N * element size.  Host-side description (see LaunchOptions).
struct PushSpec {
    uint8_t *base[8];
    size_t area_off;
    int world, rank;
    int64_t rows_per;  // a multiple of 32, so the 32 rows of an epilogue warp have one owner
};
struct FusedComm;  // peer_fused.cuh
// What a caller of quant_matmul_dispatch may ask of the launch beyond the problem itself.
struct LaunchOptions {
    int sm_reserve = 0;              // SMs the persistent kernels leave idle (a collective runs beside them)
    const PushSpec *push = nullptr;  // owners' receive areas for the output tiles (CTA-pair kernel only)
    bool push_applied = false;       // out: the launch did deliver its tiles to the owners
    const FusedComm *fused = nullptr;  // allreduce inside the CTA-pair kernel (needs push)
    bool fused_applied = false;      // out: the launch reduces and gathers the output itself
};
// Kernel-side form: one output tensor map per owner.
struct PushMaps {
    CUtensorMap m[8];
    int64_t rows_per;
    int enabled;
};

__device__ __forceinline__ float load_bias_f32(const EpilogueParams &p, int64_t n) {
    switch (p.bias_dtype) {
        case QMM_DTYPE_BF16:
            return __bfloat162float(static_cast<const __nv_bfloat16 *>(p.bias)[n]);
        case QMM_DTYPE_F16:
            return __half2float(static_cast<const __half *>(p.bias)[n]);
        case QMM_DTYPE_F32:
            return static_cast<const float *>(p.bias)[n];
        default:
            return 0.0f;
    }
}

__device__ __forceinline__ float dequant_one(int32_t acc, float scale_n, float pertoken_m, bool has_pertoken,
                                             float bias_n, bool has_bias) {
    float v = __fmul_rn(static_cast<float>(acc), scale_n);
    if (has_pertoken) v = __fmul_rn(v, pertoken_m);
    if (has_bias) v = __fadd_rn(v, bias_n);
    return v;
}

__device__ __forceinline__ int requant_one(int32_t acc, float scale_n, float pertoken_m, bool has_pertoken, float offset_n,
                                           bool has_offset) {
    return max(-128, min(127, __float2int_rn(dequant_one(acc, scale_n, pertoken_m, has_pertoken, offset_n, has_offset))));
}

// ---------------------------------------------------------------------------
// Epilogue of one warp through shared memory.
//
// The warp owns 32 accumulator rows (TMEM lanes) of a tile that is TILE_N
// columns wide.  It walks the tile in chunks whose rows are 128 bytes of
// output (128 columns of int8, 64 of bf16/f16, 32 of int32): TMEM -> registers ->
// fp32 dequantization -> a 4 KiB staging buffer laid out with the 128-byte swizzle
// (bank-conflict free 16-byte stores) -> one TMA store per chunk.  Two staging
// buffers alternate so that the store of chunk c overlaps the math of c+1.
// Outputs that break TMA's 16-byte rules (USE_TMA false at run time) leave the same
// staging row by row, a warp's lanes on consecutive columns: with every lane on a
// row of its own they took 2.9 ms at 8170 x 1952 x 23465.
// Per-column scale and bias of a chunk are fetched once per warp (coalesced)
// into a small shared array and read back as broadcasts.  Loads run one step
// ahead of their use - the next 32 columns of the accumulator and the next
// chunk's constants are under way while these columns are computed: one warp
// per scheduler has nothing else to cover them with.
// us before / now, CTA-pair kernel, M x K x N: 272 x 1024 x 28672 32.6 / 22.3,
// 2048 x 1024 x 28672 90.1 / 64.8 (int8 out 93.7 / 72.9), 2048 x 2048 x 8192 35.0 /
// 28.4; at K = 4096, where only the last tile's epilogue shows, 512 x 4096 x 28672
// 49.9 / 47.5; one-CTA kernel, 100 x 8192 x 28672 44.1 / 40.7.
//
// `stage` points to this warp's 8 KiB staging area (1024-byte aligned),
// `colbuf` to its 2*64 floats.  `chunk_counter` persists across tiles: it
// numbers the warp's TMA stores so that buffer reuse can be fenced.
// ---------------------------------------------------------------------------
template <typename OutT>
struct EpiChunk {
    static constexpr int kCols = 128 / static_cast<int>(sizeof(OutT));  // columns per 128-byte row
};

// rows of a staged chunk -> global memory, element by element
template <typename OutT>
__device__ __forceinline__ void epilogue_store_rows(const EpilogueParams &p, const uint8_t *staged, int64_t m_warp0, int64_t n0) {
    constexpr int S = static_cast<int>(sizeof(OutT)), CC = EpiChunk<OutT>::kCols;
    const int lane = threadIdx.x & 31;
    const int rows = static_cast<int>(p.M - m_warp0 < 32 ? p.M - m_warp0 : 32);
    OutT *out = static_cast<OutT *>(p.out) + m_warp0 * p.ld_out + n0;
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
#pragma unroll
        for (int i = 0; i < CC; i += 32) {
            const int byte = (i + lane) * S;
            const OutT v = *reinterpret_cast<const OutT *>(staged + r * 128 + ((((byte >> 4) ^ (r & 7))) << 4) + (byte & 15));
            if (n0 + i + lane < p.N) out[r * p.ld_out + i + lane] = v;
        }
    }
}

template <typename OutT, int TILE_N>
__device__ __forceinline__ void epilogue_warp_tile(const EpilogueParams &p, const CUtensorMap *tmap_out, bool use_tma,
                                                   uint32_t taddr_warp, int64_t m_warp0, int64_t n_tile0,
                                                   uint8_t *stage, float *colbuf, uint32_t &chunk_counter,
                                                   int64_t store_row0 = -1) {
    // store_row0: row coordinate of the warp's first row in tmap_out when that map does not start at
    // row 0 of the output (tiles pushed into another rank's receive area); -1: same as m_warp0
    constexpr int CC = EpiChunk<OutT>::kCols;
    const int lane = threadIdx.x & 31;
    const int64_t m = m_warp0 + lane;
    constexpr bool is_int = (sizeof(OutT) == 4), is_i8 = (sizeof(OutT) == 1);
    const bool has_pt = !is_int && (p.pertoken_scale != nullptr);
    const bool has_bias = (p.bias != nullptr) && (is_int || is_i8 ? p.bias_dtype == QMM_DTYPE_I32
                                                                  : (p.bias_dtype != QMM_DTYPE_NONE &&
                                                                     p.bias_dtype != QMM_DTYPE_I32));
    const float pt = (has_pt && m < p.M) ? __ldg(p.pertoken_scale + m) : 1.0f;
    const uint32_t stage_u32 = smem_u32(stage);
    if (m_warp0 >= p.M) return;  // the warp's rows are all padding

    // constants of 32 columns a word: of a chunk (16- and 32-bit outputs), or of the next 32 columns (int8)
    constexpr int kAhead = is_i8 ? 1 : CC / 32;
    float next_sc[kAhead], next_add[kAhead];  // add: bias (16-bit), int32 bias as bits (int32), offset (int8)
    int32_t next_bias = 0;                    // int8
    auto fetch = [&](int64_t first) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int64_t n = first + q * 32 + lane;
            next_sc[q] = is_i8 ? 0.0f : 1.0f;
            next_add[q] = 0.0f;
            if (is_i8) next_bias = 0;
            if (n >= p.N) continue;
            if constexpr (is_int) {
                if (has_bias) next_add[q] = __int_as_float(__ldg(static_cast<const int32_t *>(p.bias) + n));
            } else {
                next_sc[q] = p.scale_is_scalar ? __ldg(p.scale) : __ldg(p.scale + n);
                if constexpr (is_i8) {
                    if (p.offset != nullptr) next_add[q] = p.offset_is_scalar ? __ldg(p.offset) : __ldg(p.offset + n);
                    if (has_bias) next_bias = __ldg(static_cast<const int32_t *>(p.bias) + n);
                } else if (has_bias) {
                    next_add[q] = load_bias_f32(p, n);
                }
            }
        }
    };
    fetch(n_tile0);
    uint32_t ahead[32];
    tmem_ld_32x32(taddr_warp, ahead);

#pragma unroll 1
    for (int c = 0; c < TILE_N / CC; ++c) {
        const int64_t n0 = n_tile0 + static_cast<int64_t>(c) * CC;
        if (n0 >= p.N) break;
        const uint32_t buf = chunk_counter & 1;
        // the TMA store that last read this buffer (two chunks ago) must have finished reading it
        if (lane == 0) tma_store_wait_read<1>();
        __syncwarp();

        if constexpr (!is_i8) {
            // per-column constants of this chunk -> shared, as fp32 bit patterns
#pragma unroll
            for (int q = 0; q < kAhead; ++q) {
                colbuf[q * 32 + lane] = next_sc[q];
                colbuf[64 + q * 32 + lane] = next_add[q];
            }
            if (c + 1 < TILE_N / CC) fetch(n0 + CC);
            __syncwarp();
        }

        uint8_t *dst_row = stage + buf * 4096 + lane * 128;
#pragma unroll
        for (int h = 0; h < CC / 32; ++h) {
            if constexpr (is_i8) {  // scale, offset and int32 bias of 32 columns at a time
                __syncwarp();  // the previous columns' constants have been read
                colbuf[lane] = next_sc[0];
                colbuf[32 + lane] = next_add[0];
                colbuf[64 + lane] = __int_as_float(next_bias);
                if (h + 1 < CC / 32 || c + 1 < TILE_N / CC) fetch(n0 + h * 32 + 32);
                __syncwarp();
            }
            uint32_t acc[32];
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                acc[j] = ahead[j];
                asm volatile("" : "+r"(acc[j]));  // read behind the wait
            }
            if (h + 1 < CC / 32 || c + 1 < TILE_N / CC) tmem_ld_32x32(taddr_warp + c * CC + (h + 1) * 32, ahead);
            if constexpr (is_i8) {
                const bool has_off = p.offset != nullptr;
#pragma unroll
                for (int j = 0; j < 32; j += 16) {
                    uint32_t w[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 s4 = *reinterpret_cast<const float4 *>(colbuf + j + q * 4);
                        const float4 o4 = *reinterpret_cast<const float4 *>(colbuf + 32 + j + q * 4);
                        const float4 b4 = *reinterpret_cast<const float4 *>(colbuf + 64 + j + q * 4);
                        const float sv[4] = {s4.x, s4.y, s4.z, s4.w}, ov[4] = {o4.x, o4.y, o4.z, o4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
                        w[q] = 0;
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            w[q] |= (static_cast<uint32_t>(requant_one(static_cast<int32_t>(acc[j + q * 4 + t]) + __float_as_int(bv[t]), sv[t],
                                                                       pt, has_pt, ov[t], has_off)) & 0xffu) << (8 * t);
                    }
                    const int chunk16 = (h * 32 + j) / 16;
                    *reinterpret_cast<uint4 *>(dst_row + ((chunk16 ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            } else if constexpr (sizeof(OutT) == 4) {
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 b4 = *reinterpret_cast<const float4 *>(colbuf + 64 + h * 32 + j);
                    int4 v;
                    v.x = static_cast<int32_t>(acc[j + 0]) + __float_as_int(b4.x);
                    v.y = static_cast<int32_t>(acc[j + 1]) + __float_as_int(b4.y);
                    v.z = static_cast<int32_t>(acc[j + 2]) + __float_as_int(b4.z);
                    v.w = static_cast<int32_t>(acc[j + 3]) + __float_as_int(b4.w);
                    const int chunk16 = (h * 32 + j) / 4;  // 16-byte chunk index within the 128-byte row
                    *reinterpret_cast<int4 *>(dst_row + ((chunk16 ^ (lane & 7)) << 4)) = v;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                    float f[8];
#pragma unroll
                    for (int q4 = 0; q4 < 2; ++q4) {
                        const float4 s4 = *reinterpret_cast<const float4 *>(colbuf + h * 32 + j + q4 * 4);
                        const float4 b4 = *reinterpret_cast<const float4 *>(colbuf + 64 + h * 32 + j + q4 * 4);
                        f[q4 * 4 + 0] = dequant_one(static_cast<int32_t>(acc[j + q4 * 4 + 0]), s4.x, pt, has_pt, b4.x, has_bias);
                        f[q4 * 4 + 1] = dequant_one(static_cast<int32_t>(acc[j + q4 * 4 + 1]), s4.y, pt, has_pt, b4.y, has_bias);
                        f[q4 * 4 + 2] = dequant_one(static_cast<int32_t>(acc[j + q4 * 4 + 2]), s4.z, pt, has_pt, b4.z, has_bias);
                        f[q4 * 4 + 3] = dequant_one(static_cast<int32_t>(acc[j + q4 * 4 + 3]), s4.w, pt, has_pt, b4.w, has_bias);
                    }
                    uint4 w;
                    w.x = pack2<OutT>(f[0], f[1]);
                    w.y = pack2<OutT>(f[2], f[3]);
                    w.z = pack2<OutT>(f[4], f[5]);
                    w.w = pack2<OutT>(f[6], f[7]);
                    const int chunk16 = (h * 32 + j) / 8;
                    *reinterpret_cast<uint4 *>(dst_row + ((chunk16 ^ (lane & 7)) << 4)) = w;
                }
            }
        }
        if (!use_tma) {
            __syncwarp();
            epilogue_store_rows<OutT>(p, stage + buf * 4096, m_warp0, n0);
            ++chunk_counter;
            continue;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            tma_store_2d(tmap_out, stage_u32 + buf * 4096, static_cast<int32_t>(n0),
                         static_cast<int32_t>(store_row0 >= 0 ? store_row0 : m_warp0));
            tma_store_commit();
        }
        ++chunk_counter;
    }
    tmem_ld_wait();  // of a tile that ends inside the output's last columns, one load is still under way
}

// One element (used by kernels whose threads own a column of the accumulator).
template <typename OutT>
__device__ __forceinline__ void epilogue_one(const EpilogueParams &p, int64_t m, int64_t n, int32_t acc) {
    if (m >= p.M || n >= p.N) return;
    OutT *o = static_cast<OutT *>(p.out) + m * p.ld_out + n;
    if constexpr (sizeof(OutT) == 1) {
        const bool has_pt = (p.pertoken_scale != nullptr), has_off = (p.offset != nullptr);
        const float sc = p.scale_is_scalar ? __ldg(p.scale) : __ldg(p.scale + n);
        const float off = has_off ? (p.offset_is_scalar ? __ldg(p.offset) : __ldg(p.offset + n)) : 0.0f;
        const int32_t bi = p.bias != nullptr ? __ldg(static_cast<const int32_t *>(p.bias) + n) : 0;
        *o = static_cast<OutT>(requant_one(acc + bi, sc, has_pt ? __ldg(p.pertoken_scale + m) : 1.0f, has_pt, off, has_off));
    } else if constexpr (sizeof(OutT) == 4) {
        const bool has_bias = (p.bias != nullptr && p.bias_dtype == QMM_DTYPE_I32);
        *reinterpret_cast<int32_t *>(o) = acc + (has_bias ? __ldg(static_cast<const int32_t *>(p.bias) + n) : 0);
    } else {
        const bool has_bias = (p.bias != nullptr && p.bias_dtype != QMM_DTYPE_NONE && p.bias_dtype != QMM_DTYPE_I32);
        const bool has_pt = (p.pertoken_scale != nullptr);
        const float pt = has_pt ? __ldg(p.pertoken_scale + m) : 1.0f;
        const float sc = p.scale_is_scalar ? __ldg(p.scale) : __ldg(p.scale + n);
        const float bi = has_bias ? load_bias_f32(p, n) : 0.0f;
        *o = from_float<OutT>(dequant_one(acc, sc, pt, has_pt, bi, has_bias));
    }
}

}  // namespace qmm
