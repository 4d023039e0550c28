// W4A16 matmul over PREPACKED weights (npu_weight_quant_batchmatmul after a one-time layout pass).
//
// The stock layout, int32 [K, N/8] with eight neighbouring COLUMNS per word, is the wrong way round
// for every tensor-core operand format (they keep consecutive k of ONE column together), and pairing
// the rows at run time costs more integer instructions than the HBM stream leaves time for.  The
// reference has the same notion of a private matmul weight format: it casts operands from the plain
// "ND" layout to the fractal "NZ" layout around its matmul
// (op_plugin/ops/base_ops/aclops/MmKernelNpu.cpp:80-94, :301-316).  Here the format is:
//
//   block (t, c) = output columns [128 t, 128 t + 128) x k rows [128 c, 128 c + 128), 8704 bytes,
//   blocks ordered [t][c] so that a CTA's share of the work is one contiguous byte stream:
//     bytes [0, 8192)     four sub-steps of 32 k; sub-step s holds, for column r = 0..127, one
//                         16-byte vector at (s * 128 + r) * 16: word i of the vector covers
//                         k = 32 s + 8 i .. + 7 of that column, nibble j (j < 4) = k + 2 j,
//                         nibble j + 4 = k + 2 j + 1  (two's complement, as in the stock layout)
//     bytes [8192, 8448)  scale[g, n]            as 16-bit floats, g = group of the block's k rows
//     bytes [8448, 8704)  offset[g, n] * scale[g, n], rounded once to the 16-bit type
//   Columns beyond N are stored as zeros, and the number of blocks along K is rounded up to an even
//   count with an all-zero block (a stage of the kernel is a PAIR of blocks).  Requires K % 128 == 0
//   and group % 128 == 0.
//
// With that order `(word >> 4 j) & 0x000f000f` IS a tensor-memory operand column: two consecutive
// k of one output column as two 16-bit floats (after OR-ing exponent bits).  One thread owns one
// output column, so its scale and offset are scalars, and the weight
//     W = (w + offset) * scale = fma(w, scale, offset * scale)
// is finished in registers (one exact subtraction of the exponent constant, one fused multiply-add
// per pair, rounded once to the 16-bit type) and written to TENSOR MEMORY with tcgen05.st.  The MMA
// (kind::f16, 128 x Mpad x 16) takes that operand from tensor memory and the activations from
// shared memory, so the expanded weights never touch shared memory and the accumulator stays in
// tensor memory over the whole K range: no per-group pass over the accumulator, whatever M is.
//
// Warp roles (736 threads): warp 0 streams the packed weights (a stage is a pair of blocks = 17408
// contiguous bytes, one bulk copy); warp 1 streams the matching activation tiles by TMA into a ring
// of their own; warp 2 issues the MMAs (several under one election); warps 3-18 unpack
// (four teams of four warps; team s converts sub-step s of both blocks of a stage; a warp touches the
// 32 tensor-memory lanes 32 * (warp % 4)); warps 19-22 are the epilogue.  An unpack warp announces the
// operand columns of stage i only after it has converted stage i+1, so the latency of its
// tensor-memory stores hides behind the next stage's arithmetic.  A narrow form serves up to 64 token
// rows, a wide form row tiles of up to 256 (PForm).  Work is cut into contiguous ranges of (output
// tile, block pair), equal shares or whole tiles; a tile shared by several CTAs is summed from per-CTA
// slots in slot order by the CTA that arrives last, so results do not depend on arrival order.
//
// Measured bounds (B200, K = 8192, N = 28672).  Narrow: the unpack warps.  The conversion is 15
// instructions per word (the packed 16-bit ones and the logic ones issue at half rate, 64 lanes per
// clock and SM), about 1100 clocks per 256-k stage and SM where the memory needs 760: 27 us of the 37 us
// that 16 tokens take (64 tokens 38-41 us) at 66 % of the issue slots; the rest is start, last sums and
// hand-offs between the roles.  An MMA of these sizes takes about 17 clocks when eight are issued under one
// election with uniform operands; with the role index not known to be warp-uniform the MMA warp spent
// 75 clocks on each (45 / 51 us).  Wide: the tensor pipe and the power cap: 256 tokens 100 us, 2048
// tokens 733 us = 1.31 PFLOP/s of a measured 1.41 sustained.
#include "qmm_common.cuh"
#include "w4a16_gemv.cuh"
#include "w4a16_simt.cuh"

namespace qmm {

namespace {

constexpr int kPTileN = 128;                          // output columns per tile = rows of the MMA
constexpr int kPChunkK = 128;                         // k rows per block
constexpr int kPSubK = 32;                            // k rows per sub-step (one 16-byte vector per column)
constexpr int kPSubs = kPChunkK / kPSubK;             // 4
constexpr int kPWBytes = kPTileN * kPChunkK / 2;      // 8192
constexpr int kPSOBytes = 2 * kPTileN * 2;            // 512: scale, offset * scale
constexpr int kPBlockBytes = kPWBytes + kPSOBytes;    // 8704
constexpr int kPMaxM = 64;                            // token rows of the narrow form
constexpr int kPMaxWide = 256;                        // token rows of a tile of the wide form
constexpr int kPPair = 2;                             // blocks per stage
constexpr int kPStageK = kPPair * kPChunkK;           // 256 k rows per stage
constexpr int kPStageWBytes = kPPair * kPBlockBytes;  // 17408 bytes of packed weights per stage
constexpr int kPTeams = kPSubs;
constexpr int kPUnpackWarps = 4 * kPTeams;            // 16
constexpr int kPEpiWarps = 4;
constexpr int kPMmaWarp = 2;
constexpr int kPFirstUnpackWarp = 3;
constexpr int kPFirstEpiWarp = kPFirstUnpackWarp + kPUnpackWarps;
constexpr int kPThreads = (kPFirstEpiWarp + kPEpiWarps) * 32;  // 736
constexpr int kPMaxRing = 3;
constexpr int kPMaxXStages = 8;                       // activation tiles in shared memory
constexpr uint32_t kPRingCols = kPStageK / 2;         // 128 columns per stage: two 16-bit k per column
constexpr uint32_t kPMaxDBufs = 2;
// Two forms of the kernel.  Narrow (up to 64 token rows, weight-bandwidth bound): two accumulators in columns
// [0, 128), three stages of the operand ring behind, activation stages of 256 k.  Wide (more rows, bound by the MMAs,
// 8 * rows clocks per 256-k stage, from about 140 rows on; by the unpack warps below that): one accumulator of up to
// 256 columns, two ring stages, activation stages of 64 k, since a tile of 256 rows x 256 k alone is 128 KiB.
template <bool WIDE>
struct PForm {
    static constexpr int kTok = WIDE ? kPMaxWide : kPMaxM;
    static constexpr uint32_t kDBufs = WIDE ? 1 : 2;
    static constexpr uint32_t kACol0 = kDBufs * kTok;
    static constexpr int kRing = WIDE ? 2 : 3;
    static constexpr int kXBoxes = WIDE ? 1 : 4;      // boxes of 64 k per activation stage
    static_assert(kACol0 + kRing * kPRingCols <= 512, "tensor memory");
};
constexpr uint32_t kPTmemCols = 512;
constexpr int kPMaxStages = 8;
constexpr size_t kPCounterBytes = 64 * 1024;          // tile counters: a fixed area at the start of the scratch
constexpr size_t kPSmemBudget = 200 * 1024, kPSmemBudgetWide = 220 * 1024;
constexpr int kPWideStages = 4;                       // packed-weight stages of the wide form

struct PSmemTail {
    uint64_t w_full[kPMaxStages];   // packed weights of a stage have landed
    uint64_t w_empty[kPMaxStages];  // ... and have been read into registers by all unpack warps
    uint64_t x_full[kPMaxXStages];  // activation tile of a stage has landed
    uint64_t x_empty[kPMaxXStages]; // ... and the MMAs that read it are complete
    uint64_t a_full[kPMaxRing];        // operand columns of a ring slot are written (16 unpack warps)
    uint64_t mma_done[kPMaxRing];      // the MMAs of a ring slot are complete: its columns are free
    uint64_t tmem_full[kPMaxDBufs];
    uint64_t tmem_empty[kPMaxDBufs];
    uint32_t tmem_base;
    uint32_t abort_flag;
    uint32_t is_last;
    uint32_t epi_abort;
};

struct PParams {
    const uint8_t *packed;
    const void *bias;
    void *out;
    int64_t ld_out;
    int M, N;
    int mpad;         // token rows of a tile, a multiple of 16
    int nblk;         // tiles of token rows; an output tile is q = column tile * nblk + row tile
    int share, extra, grain;  // wide form, see p_first_item; grain = nchunks: whole output tiles, 1: equal shares of the block pairs
    int out_vec;      // rows of out meet the alignment of 8-byte stores
    int x_box_bytes;  // mpad * 128: one [mpad][64 k] activation box
    int nstages;      // packed-weight stages in shared memory
    int nxstages;     // activation tiles in shared memory
    int tiles_n;
    int nchunks;      // block PAIRS along K
    float *slots;        // [slots][mpad][128], see p_slot
    uint32_t *counters;  // [output tiles], zero between calls
    uint32_t *status;
};

__device__ __forceinline__ int p_cta_of_item(int64_t u, int64_t total, int64_t G) {
    return static_cast<int>((u * G + G - 1) / total);
}

// Four K=16 MMAs (64 k, one activation box) under one election; see mma_f16_ts_warp_x8.
__device__ __forceinline__ void p_mma_x4(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p, e, t;\n\t"
        ".reg .b64 bd;\n\t"
        ".reg .b32 a, bl;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %4, p;\n\t"
        "add.u32 a, %1, 8;\n\t"
        "add.u32 bl, %2, 2;\n\t"
        "mov.b64 bd, {bl, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], bd, %4, t;\n\t"
        "add.u32 a, %1, 16;\n\t"
        "add.u32 bl, %2, 4;\n\t"
        "mov.b64 bd, {bl, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], bd, %4, t;\n\t"
        "add.u32 a, %1, 24;\n\t"
        "add.u32 bl, %2, 6;\n\t"
        "mov.b64 bd, {bl, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], bd, %4, t;\n\t"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void pepi_bar_sync() { asm volatile("bar.sync 3, 128;" ::: "memory"); }

// (a & b) ^ c in one logic instruction
__device__ __forceinline__ uint32_t p_and_xor(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0x6a;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// (nibble ^ 8) | exponent bits = kRaw0 + 8 + w as a 16-bit float; subtracting the constant is exact.
template <typename T>
struct PMagic;
template <>
struct PMagic<__nv_bfloat16> {
    using T2 = __nv_bfloat162;
    static constexpr uint32_t kFlip = 0x43084308u;  // 128.0 | 8
    static constexpr uint32_t kFmt = 1;
    static __device__ __forceinline__ T2 bias2() { return __floats2bfloat162_rn(136.0f, 136.0f); }
};
template <>
struct PMagic<__half> {
    using T2 = __half2;
    static constexpr uint32_t kFlip = 0x64086408u;  // 1024.0 | 8
    static constexpr uint32_t kFmt = 0;
    static __device__ __forceinline__ T2 bias2() { return __floats2half2_rn(1032.0f, 1032.0f); }
};

// Items are dealt out in contiguous ranges, as even as they go.  The narrow form cuts at total * cta / CTAs: where an fp32
// sum is cut decides its last bits, so results of up to 64 tokens depend on this rule.  The wide form deals out p.share
// items, or one more for the first p.extra CTAs, times p.grain.
template <bool WIDE>
__device__ __forceinline__ int p_first_item(const PParams &p, int cta) {
    if constexpr (WIDE) return (cta * p.share + min(cta, p.extra)) * p.grain;
    return static_cast<int>(static_cast<int64_t>(p.tiles_n) * p.nchunks * cta / gridDim.x);
}
template <bool WIDE>
__device__ __forceinline__ int p_cta_of(const PParams &p, int item) {
    if constexpr (WIDE) {
        const int i = item / p.grain, edge = p.extra * (p.share + 1);
        return i < edge ? i / (p.share + 1) : p.extra + (i - edge) / p.share;
    }
    return p_cta_of_item(item, static_cast<int64_t>(p.tiles_n) * p.nchunks, gridDim.x);
}
// CTAs whose ranges overlap output tile q
template <bool WIDE>
__device__ __forceinline__ int p_slot_count(const PParams &p, int q) {
    return p_cta_of<WIDE>(p, q * p.nchunks + p.nchunks - 1) - p_cta_of<WIDE>(p, q * p.nchunks) + 1;
}

// Slot of CTA `cta`'s sums of output tile q.  A contiguous range shares at most its first and its last tile, so slots
// belong to CTAs and not to tiles: a slot for every tile took 235 MB for 1000 x 4096 x 28672 and 1.88 GB for 8192 rows.
// With T tiles for G CTAs, G + min(T, G) slots are enough.  T >= G: a range begins at or behind tile `cta`, the minimum
// is cta + 0 or 1, two slots for every CTA.  T < G: it begins at or before tile `cta`, the minimum is q, and cta + q
// grows from one (CTA, tile) pair to the next.
template <bool WIDE>
__device__ __forceinline__ int p_slot(const PParams &p, int cta, int q) {
    return cta + min(q, cta + (p_first_item<WIDE>(p, cta) < q * p.nchunks ? 1 : 0));
}

// Adds the sums of tile q by its `nslots` CTAs in their order and stores the tile; thread `tid` of `threads`.  report(row): called
// for a row of the tile with a sum that is not finite (PNoReport: nothing is).
struct PNoReport {};
template <typename T, bool WIDE, typename Report>
__device__ __forceinline__ void p_add_slots(const PParams &p, int q, int nslots, int tid, int threads, const Report &report) {
    const T *bias = static_cast<const T *>(p.bias);
    const int m0 = (q % p.nblk) * p.mpad, ncol0 = (q / p.nblk) * kPTileN;
    const int vecs = min(p.mpad, p.M - m0) * (kPTileN / 4);
    const int64_t slot_vecs = static_cast<int64_t>(p.mpad) * (kPTileN / 4);
    const float4 *slots = reinterpret_cast<const float4 *>(p.slots);
    const int cta0 = p_cta_of<WIDE>(p, q * p.nchunks), slot0 = p_slot<WIDE>(p, cta0, q);
    constexpr int kElems = 2;
    for (int e0 = tid; e0 < vecs; e0 += kElems * threads) {
        float4 v[kElems];
#pragma unroll
        for (int e = 0; e < kElems; ++e) v[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int s0 = 0; s0 < nslots; s0 += 4) {
            float4 part[4][kElems];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int cta = cta0 + s0 + k;  // only the first one's range can begin before the tile
                const float4 *src = slots + (cta == cta0 ? slot0 : cta + min(q, cta)) * slot_vecs;
#pragma unroll
                for (int e = 0; e < kElems; ++e) {
                    part[k][e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (s0 + k < nslots && e0 + e * threads < vecs) part[k][e] = __ldcg(src + e0 + e * threads);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int e = 0; e < kElems; ++e) {
                    v[e].x += part[k][e].x;
                    v[e].y += part[k][e].y;
                    v[e].z += part[k][e].z;
                    v[e].w += part[k][e].w;
                }
        }
#pragma unroll
        for (int e = 0; e < kElems; ++e) {
            const int idx = e0 + e * threads;
            const int n = ncol0 + (idx % (kPTileN / 4)) * 4;
            if (idx >= vecs || n >= p.N) continue;  // N is a multiple of eight
            float f[4] = {v[e].x, v[e].y, v[e].z, v[e].w};
            if constexpr (!std::is_same<Report, PNoReport>::value) {
                if (!(isfinite(f[0]) && isfinite(f[1]) && isfinite(f[2]) && isfinite(f[3]))) report(idx / (kPTileN / 4));
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) f[k] += bias != nullptr ? to_float(bias[n + k]) : 0.0f;
            T *o = static_cast<T *>(p.out) + static_cast<int64_t>(m0 + idx / (kPTileN / 4)) * p.ld_out + n;
            if (p.out_vec) {
                *reinterpret_cast<uint2 *>(o) = make_uint2(pack2<T>(f[0], f[1]), pack2<T>(f[2], f[3]));
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) o[k] = from_float<T>(f[k]);
            }
        }
    }
}

// The calling threads have stored this CTA's sums of tile q: reports that, and if it completes the tile adds the slots
// and stores the tile.  EPILOGUE: the four epilogue warps call, otherwise the whole CTA.  Inlined: as a call with the
// parameters' address it slows the whole kernel down (34 -> 43 us for 16 tokens).
template <typename T, bool WIDE, bool EPILOGUE, typename Report = PNoReport>
__device__ __forceinline__ void p_finish_shared(const PParams &p, int q, volatile uint32_t *abort_flag, uint32_t *flag,
                                                const Report &report = Report()) {
    auto barrier = [] {
        if (EPILOGUE)
            pepi_bar_sync();
        else
            __syncthreads();
    };
    const int nslots = p_slot_count<WIDE>(p, q);
    if (nslots <= 1) return;
    const int tid = static_cast<int>(threadIdx.x) - (EPILOGUE ? kPFirstEpiWarp * 32 : 0);
    barrier();
    if (tid == 0) {
        uint32_t last = 0;
        if (*abort_flag == 0) {  // a CTA that was cut short never completes a tile
            uint32_t old;
            // release: cumulative over the CTA's slot stores, which the barrier has ordered; acquire: the others'
            asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(p.counters + q) : "memory");
            last = old + 1 == static_cast<uint32_t>(nslots) ? 1u : 0u;
            if (last) p.counters[q] = 0;
        }
        *flag = last;
    }
    barrier();
    if (*reinterpret_cast<volatile uint32_t *>(flag) != 0) p_add_slots<T, WIDE>(p, q, nslots, tid, EPILOGUE ? kPEpiWarps * 32 : kPThreads, report);
    barrier();  // the flag is written again for the next tile
}

template <typename T, bool WIDE>
__global__ void __launch_bounds__(kPThreads, 1)
w4a16_prepacked_kernel(const __grid_constant__ CUtensorMap tmap_x, PParams p) {
    using T2 = typename PMagic<T>::T2;
    using F = PForm<WIDE>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t nstages = static_cast<uint32_t>(p.nstages);
    const uint32_t x_box = static_cast<uint32_t>(p.x_box_bytes);
    const uint32_t x_slot = F::kXBoxes * x_box;   // an activation stage: boxes of [mpad][64 k]
    const uint32_t nxstages = static_cast<uint32_t>(p.nxstages);
    const uint32_t w_off = nxstages * x_slot;     // the packed-weight stages sit behind the activation tiles
    PSmemTail *tail = reinterpret_cast<PSmemTail *>(smem_aligned + w_off + nstages * kPStageWBytes);
    volatile uint32_t *abort_flag = &tail->abort_flag;

    const int warp = warp_id_uniform();
    const int lane = threadIdx.x & 31;
    // this CTA's contiguous range of (output tile, block pair) items
    const int cta = static_cast<int>(blockIdx.x);
    const int u_begin = p_first_item<WIDE>(p, cta), u_end = p_first_item<WIDE>(p, cta + 1);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < nstages; ++s) {
            mbar_init(smem_u32(&tail->w_full[s]), 1);
            mbar_init(smem_u32(&tail->w_empty[s]), kPUnpackWarps);
        }
        for (uint32_t a = 0; a < nxstages; ++a) {
            mbar_init(smem_u32(&tail->x_full[a]), 1);
            mbar_init(smem_u32(&tail->x_empty[a]), 1);
        }
        for (int a = 0; a < F::kRing; ++a) {
            mbar_init(smem_u32(&tail->a_full[a]), kPUnpackWarps);
            mbar_init(smem_u32(&tail->mma_done[a]), 1);
        }
        for (uint32_t b = 0; b < F::kDBufs; ++b) {
            mbar_init(smem_u32(&tail->tmem_full[b]), 1);
            mbar_init(smem_u32(&tail->tmem_empty[b]), kPEpiWarps);
        }
        tail->abort_flag = 0;
        tail->epi_abort = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmap_x);
    }
    if (warp == kPMmaWarp) {
        tmem_alloc(smem_u32(&tail->tmem_base), kPTmemCols);
        tmem_relinquish();
        pdl_launch_dependents();
    }
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = warp_uniform(tail->tmem_base);

    if (warp == 0) {
        // ---------------- weight producer: one bulk copy of 17408 contiguous bytes per stage ----------------
        int q = u_begin / p.nchunks, c = u_begin - q * p.nchunks;
        uint32_t st = 0, ph = 0;
        const uint32_t full0 = smem_u32(&tail->w_full[0]), empty0 = smem_u32(&tail->w_empty[0]);
        for (int it = u_begin; it < u_end; ++it) {
            if (!mbar_wait(empty0 + st * 8, ph ^ 1, abort_flag, 0x50)) break;
            if (lane == 0) {
                mbar_expect_tx(full0 + st * 8, kPStageWBytes);
                bulk_load_1d(smem_base + w_off + st * kPStageWBytes,
                             p.packed + (static_cast<int64_t>(q / p.nblk) * p.nchunks + c) * kPStageWBytes, kPStageWBytes,
                             full0 + st * 8);
            }
            __syncwarp();
            if (++st == nstages) {
                st = 0;
                ph ^= 1;
            }
            if (++c == p.nchunks) {
                c = 0;
                ++q;
            }
        }
    } else if (warp == 1) {
        // ---------------- activation producer: steps of kXBoxes boxes, 4 / kXBoxes steps an item ----------------
        constexpr int kSteps = 4 / F::kXBoxes;
        int q = u_begin / p.nchunks, k0 = (u_begin - q * p.nchunks) * kPStageK, row0 = (q % p.nblk) * p.mpad;
        const int k_end = p.nchunks * kPStageK;
        uint32_t rs = 0, rph = 0;
        for (int i = (u_end - u_begin) * kSteps; i > 0; --i) {
            if (!mbar_wait(smem_u32(&tail->x_empty[rs]), rph ^ 1, abort_flag, 0x57)) break;
            if (lane == 0) {
                const uint32_t bar = smem_u32(&tail->x_full[rs]);
                const uint32_t dst = smem_base + rs * x_slot;
                mbar_expect_tx(bar, x_slot);
#pragma unroll
                for (int b = 0; b < F::kXBoxes; ++b)  // rows beyond M and k beyond K arrive as zeros
                    tma_load_2d(dst + b * x_box, &tmap_x, k0 + b * 64, row0, bar);
            }
            __syncwarp();
            if (++rs == nxstages) {
                rs = 0;
                rph ^= 1;
            }
            k0 += F::kXBoxes * 64;
            if (k0 == k_end) {
                k0 = 0;
                ++q;
                row0 = (q % p.nblk) * p.mpad;
            }
        }
    } else if (warp == kPMmaWarp) {
        // ---------------- MMA issuer (whole warp, one elected lane issues) ----------------
        const uint32_t idesc = make_idesc(/*c=f32*/ 1, PMagic<T>::kFmt, PMagic<T>::kFmt, /*a*/ 0, /*b K-major*/ 0,
                                          kPTileN, static_cast<uint32_t>(p.mpad));
        constexpr uint32_t kDescHi = smem_desc_hi_sw128(1024);
        constexpr int kSteps = 4 / F::kXBoxes;
        const uint32_t box = x_box >> 4;
        int left = p.nchunks - u_begin % p.nchunks;  // items until the end of the output tile
        uint32_t rs = 0, rph = 0, xs = 0, xph = 0, pb = 0, pb_phase = 0, accumulate = 0, step = 0;
        for (int i = (u_end - u_begin) * kSteps; i > 0; --i) {
            if (step == 0) {
                if (accumulate == 0 && !mbar_wait(smem_u32(&tail->tmem_empty[pb]), pb_phase ^ 1, abort_flag, 0x51)) break;
                if (!mbar_wait(smem_u32(&tail->a_full[rs]), rph, abort_flag, 0x53)) break;
            }
            if (!mbar_wait(smem_u32(&tail->x_full[xs]), xph, abort_flag, 0x52)) break;
            tc_fence_after();
            const uint32_t d = tmem_base + pb * F::kTok;
            const uint32_t a = tmem_base + F::kACol0 + rs * kPRingCols;
            const uint32_t x_lo = smem_desc_lo(smem_base + xs * x_slot, 16);
            if constexpr (WIDE) {
                p_mma_x4(d, a + step * 32, x_lo, kDescHi, idesc, accumulate);
            } else {
                mma_f16_ts_warp_x8(d, a, x_lo, x_lo + box, kDescHi, idesc, accumulate);
                mma_f16_ts_warp_x8(d, a + 64, x_lo + 2 * box, x_lo + 3 * box, kDescHi, idesc, 1);
            }
            accumulate = 1;
            tc_commit_warp(smem_u32(&tail->x_empty[xs]));
            if (++xs == nxstages) {
                xs = 0;
                xph ^= 1;
            }
            if (++step < kSteps) continue;
            step = 0;
            tc_commit_warp(smem_u32(&tail->mma_done[rs]));
            if (++rs == F::kRing) {
                rs = 0;
                rph ^= 1;
            }
            if (--left == 0 || i == 1) {  // the tile's or the range's last item
                left = p.nchunks;
                tc_commit_warp(smem_u32(&tail->tmem_full[pb]));
                accumulate = 0;
                if (++pb == F::kDBufs) {
                    pb = 0;
                    pb_phase ^= 1;
                }
            }
        }
    } else if (warp < kPFirstEpiWarp) {
        // ---------------- unpack warps ----------------
        const int team = (warp - kPFirstUnpackWarp) >> 2;  // sub-step of both blocks of a stage this warp converts
        const int quarter = warp & 3;                      // tensor-memory lanes [32 quarter, +32)
        const int r = quarter * 32 + lane;                 // output column within the tile
        const uint32_t nib_mask = 0x000f000fu;
        const uint32_t flip = PMagic<T>::kFlip;
        const T2 bias2 = PMagic<T>::bias2();
        // this warp's 16 columns of sub-step `team` of block 0; block 1 is 64 columns further
        const uint32_t lane_taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + F::kACol0 + team * 16;
        uint32_t st = 0, ph = 0, rs = 0, rph = 0;
        int pending = -1;  // ring slot whose stores are in flight
        for (int it = u_begin; it < u_end; ++it) {
            if (!mbar_wait(smem_u32(&tail->w_full[st]), ph, abort_flag, 0x54)) break;
            const uint8_t *blk = smem_aligned + w_off + st * kPStageWBytes;
            uint4 wv[kPPair];
            uint32_t s32[kPPair], t32[kPPair];
#pragma unroll
            for (int b = 0; b < kPPair; ++b) {
                const uint8_t *bb = blk + b * kPBlockBytes;
                wv[b] = *reinterpret_cast<const uint4 *>(bb + (team * kPTileN + r) * 16);
                const uint32_t s16 = *reinterpret_cast<const uint16_t *>(bb + kPWBytes + r * 2);
                const uint32_t t16 = *reinterpret_cast<const uint16_t *>(bb + kPWBytes + kPTileN * 2 + r * 2);
                s32[b] = s16 * 0x10001u;
                t32[b] = t16 * 0x10001u;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tail->w_empty[st]));
            uint32_t v[kPPair][16];
#pragma unroll
            for (int b = 0; b < kPPair; ++b) {
                const T2 s2 = *reinterpret_cast<const T2 *>(&s32[b]);
                const T2 t2 = *reinterpret_cast<const T2 *>(&t32[b]);
                const uint32_t words[4] = {wv[b].x, wv[b].y, wv[b].z, wv[b].w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t raw = p_and_xor(words[i] >> (4 * j), nib_mask, flip);
                        const T2 wq = __hsub2(*reinterpret_cast<const T2 *>(&raw), bias2);  // exact: w itself
                        const T2 wf = __hfma2(wq, s2, t2);                                  // (w + offset) * scale
                        v[b][4 * i + j] = *reinterpret_cast<const uint32_t *>(&wf);
                    }
            }
            // the previous stage's stores have had this stage's arithmetic to complete: announce them
            if (pending >= 0) {
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&tail->a_full[pending]));
            }
            if (!mbar_wait(smem_u32(&tail->mma_done[rs]), rph ^ 1, abort_flag, 0x55)) break;
            tc_fence_after();
            tmem_st_32x16(lane_taddr + rs * kPRingCols, v[0]);
            tmem_st_32x16(lane_taddr + rs * kPRingCols + 64, v[1]);
            pending = static_cast<int>(rs);
            if (++rs == F::kRing) {
                rs = 0;
                rph ^= 1;
            }
            if (++st == nstages) {
                st = 0;
                ph ^= 1;
            }
        }
        if (pending >= 0) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tail->a_full[pending]));
        }
    } else {
        // ---------------- epilogue warps: thread = tensor-memory lane = one output column ----------------
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const T *bias = static_cast<const T *>(p.bias);
        T *out = static_cast<T *>(p.out);
        const int M = p.M;
        int u = u_begin;
        uint32_t pb = 0, pb_phase = 0;
        while (u < u_end) {
            const int q = u / p.nchunks;
            const int tile_begin = q * p.nchunks, tile_end = tile_begin + p.nchunks;
            const int seg_end = min(tile_end, u_end);
            const bool whole = (u == tile_begin && seg_end == tile_end);
            const int64_t n = static_cast<int64_t>(q / p.nblk) * kPTileN + row;
            const int m0 = (q % p.nblk) * p.mpad;
            const int rows = min(p.mpad, M - m0);  // token rows of this tile
            const bool n_ok = n < p.N;
            const float b = (n_ok && bias != nullptr) ? to_float(bias[n]) : 0.0f;

            if (!mbar_wait(smem_u32(&tail->tmem_full[pb]), pb_phase, abort_flag, 0x56))
                *reinterpret_cast<volatile uint32_t *>(&tail->epi_abort) = 1;
            // the four warps meet at named barriers below, so they leave together or not at all
            pepi_bar_sync();
            if (*reinterpret_cast<volatile uint32_t *>(&tail->epi_abort) != 0) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + pb * F::kTok;
            const int64_t slot_elems = static_cast<int64_t>(p.mpad) * kPTileN;
            float *mine = p.slots + p_slot<WIDE>(p, cta, q) * slot_elems + row;
            T *o = out + static_cast<int64_t>(m0) * p.ld_out + n;
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&tail->tmem_empty[pb]));
            };
            if (whole) {
                // The next 16 tokens' sums are under way while these are stored, and the accumulator is free once the last are in
                // registers: with one accumulator the tensor pipe waits for this loop.  Loading and storing in turn, 1000 x 4096 x
                // 28672 took 191-195 us and 1000 x 1024 x 28672 97; now 174 and 59 at the full clock (201 and 65 under the power cap).
                auto store = [&](const uint32_t(&v)[16], int c0) {
                    if (!n_ok) return;
                    T *at = o + static_cast<int64_t>(c0) * p.ld_out;
                    if (c0 + 16 <= rows) {  // (without this form the two take 190 and 85)
#pragma unroll
                        for (int j = 0; j < 16; ++j, at += p.ld_out) *at = from_float<T>(__uint_as_float(v[j]) + b);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j, at += p.ld_out)
                            if (c0 + j < rows) *at = from_float<T>(__uint_as_float(v[j]) + b);
                    }
                };
                auto arrived = [&](uint32_t(&v)[16], bool last) {
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) asm volatile("" : "+r"(v[j]));  // read behind the wait
                    if (last) release();
                };
                uint32_t va[16], vb[16];
                tmem_ld_32x16(taddr, va);
                for (int c0 = 0; c0 < p.mpad; c0 += 32) {
                    arrived(va, c0 + 16 >= p.mpad);
                    if (c0 + 16 < p.mpad) tmem_ld_32x16(taddr + c0 + 16, vb);
                    store(va, c0);
                    if (c0 + 16 >= p.mpad) break;
                    arrived(vb, c0 + 32 >= p.mpad);
                    if (c0 + 32 < p.mpad) tmem_ld_32x16(taddr + c0 + 32, va);
                    store(vb, c0 + 16);
                }
            } else {  // (the same here: 100 x 4096 x 4096 13.8 us, 15.0 with the longer code, which short calls fetch cold)
                for (int c0 = 0; c0 < p.mpad; c0 += 16) {
                    uint32_t v[16];
                    tmem_ld_32x16(taddr + c0, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (c0 + j < rows) __stcg(mine + (c0 + j) * kPTileN, __uint_as_float(v[j]));
                }
                release();
            }
            if (++pb == F::kDBufs) {
                pb = 0;
                pb_phase ^= 1;
            }
            // a tile that this CTA shares and leaves before the end of its range: these four warps report it, while
            // the others go on
            if (!whole && seg_end < u_end) p_finish_shared<T, WIDE, true>(p, q, abort_flag, &tail->is_last);
            u = seg_end;
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && tail->abort_flag != 0 && p.status != nullptr) atomicMax(p.status, tail->abort_flag);
    if (warp == kPMmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kPTmemCols);
    }
    // Output tiles shared with other CTAs: only the first and the last of a contiguous range can be.  The CTA that
    // arrives last adds the slots.  Most tiles are completed at the end of a range, by then with all threads, so that
    // the slots' loads of many elements are in flight together.
    if (p.grain == 1 && u_begin < u_end) p_finish_shared<T, WIDE, false>(p, (u_end - 1) / p.nchunks, abort_flag, &tail->is_last);
}

// ---- 3 to 16 token rows with the tables at hand: the weight as a whole number, scale and offset on the sums of a block ----
//
// The narrow form's unpack warps finish a weight with a multiply-add, which rounds it to 16 bits.  With few token rows that can be
// left to the sums: the operand is w itself, every block of 128 k has an accumulator of its own, and the epilogue warps fold
// it into fp32 running outputs:
//     y[m, n] += scale * acc[m, n] + scale * offset * xs[m],    xs[m] = the block's sum of x[m, :].
// The weight is never rounded, and scale and offset come from the caller's tables in full.  (An operand of w + 24 saves the
// subtraction, but its sums hold 24 times the sum of x as well: a block with one large activation loses the small ones.)
// Infinite activations make sums that are no numbers, and very large ones sums that leave fp32 where the output, which is scaled,
// would not: what is not finite is computed again, plainly (b_plain_tiles).
//
// A stage holds the nibbles of two blocks (not the stream's own tables) and their rows of scale and offset.  The epilogue warps
// also make xs, from the activation tile in shared memory: warp e takes block e / 2 and eight tokens, a lane a quarter of the
// block's k.  Everything else (roles, rings, cuts, slots) is as in the kernel above.
//
// us, this / the narrow form above / the stock layout (M x K x N): 8 x 1024 x 1024 5.7 / 5.5 / 17.2, 8 x 8192 x 1024 9.1 / 8.1 / 92,
// 8 x 4096 x 4096 10.7 / 8.9 / 33.4, 8 x 8192 x 8192 19.0 / 15.4 / 30.9, 8 x 8192 x 28672 48.4 / 33.5 / 38.8 (with w + 24 as the operand
// 5.8, 9.3, 10.4, 18.5 and 46.3; two fp32 operations an instruction in the epilogue save 1 to 3 %).  A stage takes about
// 1800 clocks, of which the epilogue warps' chain of instructions takes nearly all (waits are short, the issue slots 52 % used).
// Measured without gain: two sets of epilogue warps in turn (44-48 us for the last), sums of x by warps of their own with a ring for
// the tables (48-52), and sums of x from a kernel in front, without which the chain is half as long (42.8, but 6.5 for the first).
constexpr int kBTok = 16;
constexpr uint32_t kBAccBufs = 4;              // accumulators of a stage: two blocks x 16 columns
constexpr uint32_t kBAccCols = kPPair * kBTok;
constexpr uint32_t kBACol0 = kBAccBufs * kBAccCols;
constexpr int kBRing = 3;
static_assert(kBACol0 + kBRing * kPRingCols <= 512, "tensor memory");
constexpr int kBTableBytes = kPTileN * 2;                                     // a block's row of scale, or of offset
constexpr int kBStageBytes = kPPair * (kPWBytes + 2 * kBTableBytes);          // 17408: nibbles, nibbles, scales, offsets
static_assert(kBStageBytes == kPStageWBytes, "the plan's stages");

struct BSmemTail {
    uint64_t w_full[kPMaxStages];
    uint64_t w_empty[kPMaxStages];   // the unpack and the epilogue warps
    uint64_t x_full[kPMaxXStages];
    uint64_t x_empty[kPMaxXStages];  // the MMAs and the four epilogue warps
    uint64_t a_full[kBRing];
    uint64_t mma_done[kBRing];
    uint64_t acc_full[kBAccBufs];
    uint64_t acc_empty[kBAccBufs];
    uint32_t tmem_base;
    uint32_t abort_flag;
    uint32_t is_last;
    uint32_t epi_abort[2];           // [stage parity]: an epilogue warp gave up at that stage
    uint32_t bad_rows, bad_tiles;    // with sums that are not finite, see b_plain_tiles
    __align__(16) float xs[2][kPPair][kBTok];  // [stage parity][block][token], read four at a time
};

struct BTables {
    const void *scale, *offset;      // [groups][N]; offset may be null
    int group_blocks;                // blocks of 128 k in a group
    int nblocks;                     // blocks of 128 k along K
    const void *x;
    int64_t ld_x;
};

// The products of eight k, a word of a column and their activations, added to y.  NONFINITE: those of the activations that are not
// finite alone.
template <typename T, bool NONFINITE>
__device__ __forceinline__ float b_plain_step(float y, const uint4 &x, uint32_t word, float s, float o) {
    const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int w = static_cast<int>(word << (28 - 4 * ((e >> 1) + (e & 1) * 4))) >> 28;
        const unsigned short bits = static_cast<unsigned short>(xw[e >> 1] >> (16 * (e & 1)));
        const float v = to_float(*reinterpret_cast<const T *>(&bits));
        if (!NONFINITE || !isfinite(v)) y = fmaf(v, (static_cast<float>(w) + o) * s, y);
    }
    return y;
}
// whether any (NAN_ONLY: any NaN) of eight activations is not finite
template <typename T, bool NAN_ONLY>
__device__ __forceinline__ bool b_any_not_finite(const uint4 &x) {
    constexpr uint32_t kInf = std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u;
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    bool any = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t lo = w[j] & 0x7fffu, hi = w[j] >> 16 & 0x7fffu;
        any = any || (NAN_ONLY ? lo > kInf || hi > kInf : lo >= kInf || hi >= kInf);
    }
    return any;
}

// The bit of tile q of a CTA whose tiles are q0 .. q1: the last one, which another CTA may finish, has one of its own.
__device__ __forceinline__ uint32_t b_tile_bit(int q, int q0, int q1) { return 1u << (q == q1 ? 31 : min(q - q0, 30)); }

// Outputs whose sums are not finite, by the definition: rows (a bit each) of tiles (b_tile_bit), as the CTA has stored them.  By the whole CTA, behind its work: in the epilogue this code costs the main loop registers
// (8 x 8192 x 8192: 19.0 us, 19.5 with a call there, 22.0 with a longer function), and a thread with all of K for itself is slow.  us, operator,
// 8 x 4096 x 4096, finite 18: a NaN in every row 440 -> 23, an infinity in one 347 -> 20, 43 in every row 440 -> 70, sums of one row that leave
// fp32 347 -> 41; 8 x 28672 x 768, finite 21: 2952 -> 36, 2308 -> 30, 2953 -> 94, 2309 -> 168.  A NaN among the activations is one among the sums already; infinite activations decide alone, so only their
// products are added; where all are finite, sums left fp32, and five groups of 128 threads share K.  The scratch: 5 x 128 floats.
template <typename T>
__device__ __forceinline__ void b_plain_tiles(const PParams &p, const BTables &t, uint32_t rows, uint32_t tiles, int q0, int q1, float *part) {
    constexpr int kGroups = kPThreads / kPTileN, kVecs = kPChunkK / 8;  // vectors of eight k of a block
    const int r = threadIdx.x % kPTileN, group = threadIdx.x / kPTileN, lane = threadIdx.x & 31;
    const int vecs = t.nblocks * kVecs;
    for (; rows != 0; rows &= rows - 1) {
        const int m = __ffs(static_cast<int>(rows)) - 1;
        const uint4 *xv = reinterpret_cast<const uint4 *>(static_cast<const T *>(t.x) + m * t.ld_x);
        bool nan = false, inf = false;
        for (int v = threadIdx.x; v < vecs; v += kPThreads) {
            const uint4 x = __ldg(xv + v);
            nan = nan || b_any_not_finite<T, true>(x);
            inf = inf || b_any_not_finite<T, false>(x);
        }
        if (__syncthreads_or(nan)) continue;
        const bool infinite = __syncthreads_or(inf);
        for (int q = q0; q <= q1; ++q) {
            if ((tiles & b_tile_bit(q, q0, q1)) == 0) continue;
            const int64_t n = static_cast<int64_t>(q) * kPTileN + r;
            T *out = static_cast<T *>(p.out) + m * p.ld_out + n;
            unsigned short stored = 0;
            if (group < kGroups && n < p.N) stored = __ldcg(reinterpret_cast<const unsigned short *>(out));
            const bool wanted = group < kGroups && n < p.N && !isfinite(to_float(*reinterpret_cast<const T *>(&stored)));
            if (!__syncthreads_or(wanted)) continue;
            float y = 0.0f, s = 0.0f, o = 0.0f;
            auto load_tables = [&](int blk) {
                const int64_t at = static_cast<int64_t>(blk / t.group_blocks) * p.N + min(n, static_cast<int64_t>(p.N) - 1);
                s = to_float(static_cast<const T *>(t.scale)[at]);
                o = t.offset != nullptr ? to_float(static_cast<const T *>(t.offset)[at]) : 0.0f;
            };
            const uint8_t *stream = p.packed + static_cast<int64_t>(q) * p.nchunks * kPStageWBytes + r * 16;
            if (group < kGroups) {
                const int first = t.nblocks * group / kGroups, end = t.nblocks * (group + 1) / kGroups;
                if (infinite) {
                    bool decided = false;  // every output of the warp is a NaN already
                    for (int v0 = first * kVecs; v0 < end * kVecs && !decided; v0 += 32) {
                        const bool hit = v0 + lane < end * kVecs && b_any_not_finite<T, false>(__ldg(xv + v0 + lane));
                        for (unsigned hits = __ballot_sync(0xffffffffu, hit); hits != 0; hits &= hits - 1) {
                            const int v = v0 + __ffs(static_cast<int>(hits)) - 1, blk = v / kVecs, i = v % kVecs;
                            load_tables(blk);
                            const uint8_t *words = stream + static_cast<int64_t>(blk) * kPBlockBytes + (i >> 2) * kPTileN * 16;
                            y = b_plain_step<T, true>(y, __ldg(xv + v), __ldg(reinterpret_cast<const uint32_t *>(words) + (i & 3)), s, o);
                            decided = __all_sync(0xffffffffu, !wanted || isnan(y));
                            if (decided) break;
                        }
                    }
                } else {
                    for (int blk = first; blk < end; ++blk) {
                        load_tables(blk);
#pragma unroll 1
                        for (int sub = 0; sub < kPChunkK / kPSubK; ++sub) {
                            const uint4 w = __ldg(reinterpret_cast<const uint4 *>(stream + static_cast<int64_t>(blk) * kPBlockBytes) + sub * kPTileN);
                            const uint4 *at = xv + blk * kVecs + sub * 4;
                            y = b_plain_step<T, false>(y, __ldg(at), w.x, s, o);
                            y = b_plain_step<T, false>(y, __ldg(at + 1), w.y, s, o);
                            y = b_plain_step<T, false>(y, __ldg(at + 2), w.z, s, o);
                            y = b_plain_step<T, false>(y, __ldg(at + 3), w.w, s, o);
                        }
                    }
                }
                part[group * kPTileN + r] = y;
            }
            __syncthreads();
            if (group == 0 && wanted) {
                for (int g = 1; g < kGroups; ++g) y += part[g * kPTileN + r];
                *out = from_float<T>(y + (p.bias != nullptr ? to_float(static_cast<const T *>(p.bias)[n]) : 0.0f));
            }
            __syncthreads();
        }
    }
}

template <typename T>
__device__ __forceinline__ void b_add_words(float2 &s, const uint4 &v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const T *h = reinterpret_cast<const T *>(&w[i]);
        s = add2(s, make_float2(to_float(h[0]), to_float(h[1])));
    }
}

template <typename T>
__global__ void __launch_bounds__(kPThreads, 1)
w4a16_block_kernel(const __grid_constant__ CUtensorMap tmap_x, PParams p, BTables t) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t nstages = static_cast<uint32_t>(p.nstages), nxstages = static_cast<uint32_t>(p.nxstages);
    constexpr uint32_t kXBox = kBTok * 128, kXSlot = 4 * kXBox;  // an activation stage: four boxes of [16 tokens][64 k]
    const uint32_t w_off = nxstages * kXSlot;
    BSmemTail *tail = reinterpret_cast<BSmemTail *>(smem_aligned + w_off + nstages * kPStageWBytes);
    volatile uint32_t *abort_flag = &tail->abort_flag;

    const int warp = warp_id_uniform();
    const int lane = threadIdx.x & 31;
    const int cta = static_cast<int>(blockIdx.x);
    const int u_begin = p_first_item<false>(p, cta), u_end = p_first_item<false>(p, cta + 1);
    const auto report = [&](int q, uint32_t rows) {
        atomicOr(&tail->bad_rows, rows);
        atomicOr(&tail->bad_tiles, b_tile_bit(q, u_begin / p.nchunks, (u_end - 1) / p.nchunks));
    };

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < nstages; ++s) {
            mbar_init(smem_u32(&tail->w_full[s]), 1);
            mbar_init(smem_u32(&tail->w_empty[s]), kPUnpackWarps + kPEpiWarps);
        }
        for (uint32_t a = 0; a < nxstages; ++a) {
            mbar_init(smem_u32(&tail->x_full[a]), 1);
            mbar_init(smem_u32(&tail->x_empty[a]), 1 + kPEpiWarps);
        }
        for (int a = 0; a < kBRing; ++a) {
            mbar_init(smem_u32(&tail->a_full[a]), kPUnpackWarps);
            mbar_init(smem_u32(&tail->mma_done[a]), 1);
        }
        for (uint32_t b = 0; b < kBAccBufs; ++b) {
            mbar_init(smem_u32(&tail->acc_full[b]), 1);
            mbar_init(smem_u32(&tail->acc_empty[b]), kPEpiWarps);
        }
        tail->abort_flag = 0;
        tail->epi_abort[0] = tail->epi_abort[1] = 0;
        tail->bad_rows = tail->bad_tiles = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmap_x);
    }
    if (warp == kPMmaWarp) {
        tmem_alloc(smem_u32(&tail->tmem_base), kPTmemCols);
        tmem_relinquish();
        pdl_launch_dependents();
    }
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = warp_uniform(tail->tmem_base);

    if (warp == 0) {
        // ---------------- weight producer ----------------
        int q = u_begin / p.nchunks, c = u_begin - q * p.nchunks;
        uint32_t st = 0, ph = 0;
        const uint32_t full0 = smem_u32(&tail->w_full[0]), empty0 = smem_u32(&tail->w_empty[0]);
        for (int it = u_begin; it < u_end; ++it) {
            if (!mbar_wait(empty0 + st * 8, ph ^ 1, abort_flag, 0x70)) break;
            if (lane == 0) {
                const uint32_t dst = smem_base + w_off + st * kBStageBytes, bar = full0 + st * 8;
                // columns of this tile that exist: a multiple of eight, so the rows' copies are of whole 16 bytes
                const uint32_t cols = static_cast<uint32_t>(min(kPTileN, p.N - q * kPTileN)) * 2;
                const int blocks = min(kPPair, t.nblocks - c * kPPair);  // the last stage's second block may be padding
                mbar_expect_tx(bar, kPPair * kPWBytes + blocks * cols * (t.offset != nullptr ? 2 : 1));
                const uint8_t *src = p.packed + (static_cast<int64_t>(q) * p.nchunks + c) * kPStageWBytes;
                for (int b = 0; b < kPPair; ++b) bulk_load_1d(dst + b * kPWBytes, src + b * kPBlockBytes, kPWBytes, bar);
                for (int b = 0; b < blocks; ++b) {
                    const int64_t at = (static_cast<int64_t>((c * kPPair + b) / t.group_blocks) * p.N + static_cast<int64_t>(q) * kPTileN) * 2;
                    const uint32_t to = dst + kPPair * kPWBytes + b * kBTableBytes;
                    bulk_load_1d(to, static_cast<const uint8_t *>(t.scale) + at, cols, bar);
                    if (t.offset != nullptr) bulk_load_1d(to + kPPair * kBTableBytes, static_cast<const uint8_t *>(t.offset) + at, cols, bar);
                }
            }
            __syncwarp();
            if (++st == nstages) {
                st = 0;
                ph ^= 1;
            }
            if (++c == p.nchunks) {
                c = 0;
                ++q;
            }
        }
    } else if (warp == 1) {
        // ---------------- activation producer ----------------
        int c = u_begin % p.nchunks;
        uint32_t rs = 0, rph = 0;
        for (int it = u_begin; it < u_end; ++it) {
            if (!mbar_wait(smem_u32(&tail->x_empty[rs]), rph ^ 1, abort_flag, 0x77)) break;
            if (lane == 0) {
                const uint32_t bar = smem_u32(&tail->x_full[rs]);
                mbar_expect_tx(bar, kXSlot);
#pragma unroll
                for (int b = 0; b < 4; ++b)  // rows beyond M and k beyond K arrive as zeros
                    tma_load_2d(smem_base + rs * kXSlot + b * kXBox, &tmap_x, c * kPStageK + b * 64, 0, bar);
            }
            __syncwarp();
            if (++rs == nxstages) {
                rs = 0;
                rph ^= 1;
            }
            if (++c == p.nchunks) c = 0;
        }
    } else if (warp == kPMmaWarp) {
        // ---------------- MMA issuer: two accumulators a stage ----------------
        const uint32_t idesc = make_idesc(/*c=f32*/ 1, PMagic<T>::kFmt, PMagic<T>::kFmt, /*a*/ 0, /*b K-major*/ 0, kPTileN, kBTok);
        constexpr uint32_t kDescHi = smem_desc_hi_sw128(1024);
        constexpr uint32_t kBox = kXBox >> 4;
        uint32_t rs = 0, rph = 0, xs = 0, xph = 0, ab = 0, aph = 0;
        for (int it = u_begin; it < u_end; ++it) {
            if (!mbar_wait(smem_u32(&tail->acc_empty[ab]), aph ^ 1, abort_flag, 0x71)) break;
            if (!mbar_wait(smem_u32(&tail->x_full[xs]), xph, abort_flag, 0x72)) break;
            if (!mbar_wait(smem_u32(&tail->a_full[rs]), rph, abort_flag, 0x73)) break;
            tc_fence_after();
            const uint32_t d = tmem_base + ab * kBAccCols;
            const uint32_t a = tmem_base + kBACol0 + rs * kPRingCols;
            const uint32_t x_lo = smem_desc_lo(smem_base + xs * kXSlot, 16);
            mma_f16_ts_warp_x8(d, a, x_lo, x_lo + kBox, kDescHi, idesc, 0);
            mma_f16_ts_warp_x8(d + kBTok, a + 64, x_lo + 2 * kBox, x_lo + 3 * kBox, kDescHi, idesc, 0);
            tc_commit_warp(smem_u32(&tail->acc_full[ab]));
            tc_commit_warp(smem_u32(&tail->x_empty[xs]));
            tc_commit_warp(smem_u32(&tail->mma_done[rs]));
            if (++xs == nxstages) {
                xs = 0;
                xph ^= 1;
            }
            if (++rs == kBRing) {
                rs = 0;
                rph ^= 1;
            }
            if (++ab == kBAccBufs) {
                ab = 0;
                aph ^= 1;
            }
        }
    } else if (warp < kPFirstEpiWarp) {
        // ---------------- unpack warps ----------------
        const int team = (warp - kPFirstUnpackWarp) >> 2;
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        using T2 = typename PMagic<T>::T2;
        const T2 bias2 = PMagic<T>::bias2();
        const uint32_t lane_taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + kBACol0 + team * 16;
        uint32_t st = 0, ph = 0, rs = 0, rph = 0;
        int pending = -1;  // ring slot whose stores are in flight
        for (int it = u_begin; it < u_end; ++it) {
            if (!mbar_wait(smem_u32(&tail->w_full[st]), ph, abort_flag, 0x74)) break;
            const uint8_t *blk = smem_aligned + w_off + st * kBStageBytes;
            uint4 wv[kPPair];
#pragma unroll
            for (int b = 0; b < kPPair; ++b) wv[b] = *reinterpret_cast<const uint4 *>(blk + b * kPWBytes + (team * kPTileN + r) * 16);
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tail->w_empty[st]));
            uint32_t v[kPPair][16];
#pragma unroll
            for (int b = 0; b < kPPair; ++b) {
                const uint32_t words[4] = {wv[b].x, wv[b].y, wv[b].z, wv[b].w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t raw = p_and_xor(words[i] >> (4 * j), 0x000f000fu, PMagic<T>::kFlip);
                        const T2 wq = __hsub2(*reinterpret_cast<const T2 *>(&raw), bias2);  // exact: w itself
                        v[b][4 * i + j] = *reinterpret_cast<const uint32_t *>(&wq);
                    }
            }
            // the previous stage's stores have had this stage's arithmetic to complete: announce them
            if (pending >= 0) {
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&tail->a_full[pending]));
            }
            if (!mbar_wait(smem_u32(&tail->mma_done[rs]), rph ^ 1, abort_flag, 0x75)) break;
            tc_fence_after();
            tmem_st_32x16(lane_taddr + rs * kPRingCols, v[0]);
            tmem_st_32x16(lane_taddr + rs * kPRingCols + 64, v[1]);
            pending = static_cast<int>(rs);
            if (++rs == kBRing) {
                rs = 0;
                rph ^= 1;
            }
            if (++st == nstages) {
                st = 0;
                ph ^= 1;
            }
        }
        if (pending >= 0) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tail->a_full[pending]));
        }
    } else {
        // ---------------- epilogue warps: thread = tensor-memory lane = one output column ----------------
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const int ew = warp - kPFirstEpiWarp;
        const T *bias = static_cast<const T *>(p.bias);
        T *out = static_cast<T *>(p.out);
        const int M = p.M;
        // its share of xs: block ew / 2 of a stage, token 8 * (ew % 2) + lane % 8, k quarter lane / 8
        const int xb = ew >> 1, xtok = 8 * (ew & 1) + (lane & 7), xq = lane >> 3;
        const uint32_t x_row = (2 * xb + (xq >> 1)) * kXBox + xtok * 128;
        int u = u_begin;
        uint32_t ab = 0, aph = 0, xst = 0, xph = 0, wst = 0, wph = 0, parity = 0;
        bool ok = true;
        while (u < u_end && ok) {
            const int q = u / p.nchunks;
            const int tile_begin = q * p.nchunks, tile_end = tile_begin + p.nchunks;
            const int seg_end = min(tile_end, u_end);
            const bool whole = (u == tile_begin && seg_end == tile_end);
            const int64_t n = static_cast<int64_t>(q) * kPTileN + row;
            const bool n_ok = n < p.N;
            const float b = (n_ok && bias != nullptr) ? to_float(bias[n]) : 0.0f;
            float2 y[kBTok / 2];  // of two tokens
#pragma unroll
            for (int j = 0; j < kBTok / 2; ++j) y[j] = make_float2(0.0f, 0.0f);
            auto output = [&](int j) { return j & 1 ? y[j >> 1].y : y[j >> 1].x; };
            for (int it = u; it < seg_end; ++it) {
                ok = mbar_wait(smem_u32(&tail->x_full[xst]), xph, abort_flag, 0x78);
                float2 sums = make_float2(0.0f, 0.0f);
                const uint8_t *xr = smem_aligned + xst * kXSlot + x_row;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    b_add_words<T>(sums, *reinterpret_cast<const uint4 *>(xr + (((4 * (xq & 1) + c) ^ (xtok & 7)) << 4)));
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&tail->x_empty[xst]));
                float sum = sums.x + sums.y;
                sum += __shfl_xor_sync(0xffffffffu, sum, 8);
                sum += __shfl_xor_sync(0xffffffffu, sum, 16);
                if (lane < 8) tail->xs[parity][xb][xtok] = sum;
                // scale and scale * offset of the stage's two blocks
                ok = ok && mbar_wait(smem_u32(&tail->w_full[wst]), wph, abort_flag, 0x79);
                float sc[kPPair], tc[kPPair];
                const T *table = reinterpret_cast<const T *>(smem_aligned + w_off + wst * kBStageBytes + kPPair * kPWBytes) + row;
#pragma unroll
                for (int k = 0; k < kPPair; ++k) {
                    const bool real = n_ok && (it - tile_begin) * kPPair + k < t.nblocks;
                    sc[k] = real ? to_float(table[k * kPTileN]) : 0.0f;
                    tc[k] = real && t.offset != nullptr ? sc[k] * to_float(table[(kPPair + k) * kPTileN]) : 0.0f;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&tail->w_empty[wst]));
                ok = ok && mbar_wait(smem_u32(&tail->acc_full[ab]), aph, abort_flag, 0x76);
                // the four warps meet at named barriers, so they leave together or not at all
                volatile uint32_t *gave_up = &tail->epi_abort[parity];
                if (!ok) *gave_up = 1;
                pepi_bar_sync();
                if (*gave_up != 0) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + ab * kBAccCols;
                uint32_t v[kPPair][16];
                tmem_ld_32x16(taddr, v[0]);
                tmem_ld_32x16(taddr + kBTok, v[1]);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&tail->acc_empty[ab]));
#pragma unroll
                for (int k = 0; k < kPPair; ++k)
#pragma unroll
                    for (int j = 0; j < kBTok; j += 4) {
                        if (j >= M) break;
                        const float4 x4 = *reinterpret_cast<const float4 *>(&tail->xs[parity][k][j]);
                        const float2 sc2 = make_float2(sc[k], sc[k]), tc2 = make_float2(tc[k], tc[k]);
                        auto fold = [&](float2 &to, float2 xs, uint32_t a0, uint32_t a1) {
                            to = fma2(tc2, xs, fma2(sc2, make_float2(__uint_as_float(a0), __uint_as_float(a1)), to));
                        };
                        fold(y[j / 2], make_float2(x4.x, x4.y), v[k][j], v[k][j + 1]);
                        fold(y[j / 2 + 1], make_float2(x4.z, x4.w), v[k][j + 2], v[k][j + 3]);
                    }
                parity ^= 1;
                if (++wst == nstages) {
                    wst = 0;
                    wph ^= 1;
                }
                if (++xst == nxstages) {
                    xst = 0;
                    xph ^= 1;
                }
                if (++ab == kBAccBufs) {
                    ab = 0;
                    aph ^= 1;
                }
            }
            if (!ok) break;
            if (whole) {
                if (n_ok) {
                    uint32_t again = 0;
#pragma unroll
                    for (int j = 0; j < kBTok; ++j) {
                        if (j >= M) break;
                        again |= !isfinite(output(j)) ? 1u << j : 0u;
                        out[static_cast<int64_t>(j) * p.ld_out + n] = from_float<T>(output(j) + b);
                    }
                    if (again != 0) report(q, again);
                }
            } else {
                float *mine = p.slots + p_slot<false>(p, cta, q) * (static_cast<int64_t>(p.mpad) * kPTileN) + row;
#pragma unroll
                for (int j = 0; j < kBTok; ++j)
                    if (j < M) __stcg(mine + j * kPTileN, output(j));
                if (seg_end < u_end) p_finish_shared<T, false, true>(p, q, abort_flag, &tail->is_last, [&](int j) { report(q, 1u << j); });
            }
            u = seg_end;
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && tail->abort_flag != 0 && p.status != nullptr) atomicMax(p.status, tail->abort_flag);
    if (warp == kPMmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kPTmemCols);
    }
    if (u_begin < u_end) {
        const int q1 = (u_end - 1) / p.nchunks;
        p_finish_shared<T, false, false>(p, q1, abort_flag, &tail->is_last, [&](int j) { report(q1, 1u << j); });
        const uint32_t rows = *static_cast<volatile uint32_t *>(&tail->bad_rows), tiles = *static_cast<volatile uint32_t *>(&tail->bad_tiles);
        if (rows != 0 && *abort_flag == 0) b_plain_tiles<T>(p, t, rows, tiles, u_begin / p.nchunks, q1, reinterpret_cast<float *>(smem_aligned));
    }
}

// ---- layout pass and its inverse ----------------------------------------------------------------------

// Eight words of one word column, of rows k .. k + 7, to the eight columns' words: nibble j of row e becomes the nibble of row e
// in word j, in the block's order of rows (0, 2, 4, 6, 1, 3, 5, 7).  A transposition by halves, bytes and nibbles.
__device__ __forceinline__ void p_transpose8(uint32_t (&w)[8]) {
    const uint32_t b[8] = {w[0], w[2], w[4], w[6], w[1], w[3], w[5], w[7]};
    uint32_t x[8], y[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[i] = __byte_perm(b[i], b[i + 4], 0x5410);
        x[i + 4] = __byte_perm(b[i], b[i + 4], 0x7632);
    }
#pragma unroll
    for (int h = 0; h < 8; h += 4)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            y[h + i] = __byte_perm(x[h + i], x[h + i + 2], 0x6240);      // columns h, h + 1
            y[h + i + 2] = __byte_perm(x[h + i], x[h + i + 2], 0x7351);  // columns h + 2, h + 3
        }
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        w[j] = (y[j] & 0x0f0f0f0fu) | ((y[j + 1] & 0x0f0f0f0fu) << 4);
        w[j + 1] = ((y[j] >> 4) & 0x0f0f0f0fu) | (y[j + 1] & 0xf0f0f0f0u);
    }
}

// One CTA per chunk of 128 k and TILES tiles: rows of 256 (64) bytes come in, are transposed in registers and leave as four (one)
// blocks, through one buffer in shared memory both ways.  With a load from global memory for every nibble (a thread a 16-byte
// vector, 32 strided loads each) 8192 x 28672 took 128 us, 4096 x 4096 7.2 and 1024 x 1024 2.7; now 65, 5.7 and 2.0.  One tile a CTA
// where four leave SMs without work (1024 x 1024: 3.9 with four).  A weight's first call pays for this pass, and every call of three to eight rows that
// the operator sends here.
constexpr int kPPackThreads = 256;
template <typename T, int TILES>
__global__ void __launch_bounds__(kPPackThreads)
w4a16_prepack_kernel(const int32_t *__restrict__ w, int64_t ld_w, int aligned, const T *__restrict__ scale,
                     const T *__restrict__ offset, int64_t group, int64_t N, int64_t K, int nchunks,
                     uint8_t *__restrict__ out) {
    constexpr int kWords = TILES * kPTileN / 8;  // packed words of a row
    constexpr int kSwap = TILES > 1 ? 3 : 1;
    __shared__ __align__(16) uint32_t buf[kPChunkK * kWords];
    const int c = blockIdx.x;  // runs over the padded (even) number of blocks
    const int64_t tile0 = static_cast<int64_t>(blockIdx.y) * TILES, word0 = tile0 * (kPTileN / 8), words = N / 8;
    const int64_t k0 = static_cast<int64_t>(c) * kPChunkK;
    const bool real = k0 < K;  // the padding block and the padding columns are zeros
    pdl_launch_dependents();
    pdl_wait();
    // word i of row k lies at i ^ 8 (k / 8 % 4): lanes that read four groups of eight rows find them in different banks (in rows
    // of one tile, whose 16 words allow only % 2, in pairs of banks)
    for (int v = threadIdx.x; v < kPChunkK * kWords / 4; v += kPPackThreads) {
        const int k = v / (kWords / 4), i = v % (kWords / 4) * 4;
        const int32_t *src = w + (k0 + k) * ld_w + word0 + i;
        uint4 q = make_uint4(0, 0, 0, 0);
        if (real && aligned && word0 + i + 4 <= words) {
            q = __ldg(reinterpret_cast<const uint4 *>(src));
        } else if (real) {
            if (word0 + i < words) q.x = static_cast<uint32_t>(src[0]);
            if (word0 + i + 1 < words) q.y = static_cast<uint32_t>(src[1]);
            if (word0 + i + 2 < words) q.z = static_cast<uint32_t>(src[2]);
            if (word0 + i + 3 < words) q.w = static_cast<uint32_t>(src[3]);
        }
        *reinterpret_cast<uint4 *>(buf + k * kWords + (i ^ ((k >> 3 & kSwap) << 3))) = q;
    }
    __syncthreads();
    // a lane: word i of the 16-byte vectors (eight rows) and one of eight word columns; a warp: TILES of their 8 TILES places
    const int lane = threadIdx.x & 31, i = lane & 3;
    uint32_t t[TILES][8];
#pragma unroll
    for (int q = 0; q < TILES; ++q) {
        const int place = (threadIdx.x >> 5) * TILES + q, s = place & 3, col = (place >> 2) * 8 + (lane >> 2);
#pragma unroll
        for (int e = 0; e < 8; ++e) t[q][e] = buf[((s * 4 + i) * 8 + e) * kWords + (col ^ ((i & kSwap) << 3))];
        p_transpose8(t[q]);
    }
    __syncthreads();
    // vector v of a block lies at v ^ (v / 8 % 8)
#pragma unroll
    for (int q = 0; q < TILES; ++q) {
        const int place = (threadIdx.x >> 5) * TILES + q, s = place & 3, col = (place >> 2) * 8 + (lane >> 2);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int v = s * kPTileN + (col & 15) * 8 + j;
            buf[((col >> 4) * (kPWBytes / 16) + (v ^ (v >> 3 & 7))) * 4 + i] = t[q][j];
        }
    }
    __syncthreads();
    const int64_t tiles = (N + kPTileN - 1) / kPTileN;
    for (int v = threadIdx.x; v < TILES * (kPWBytes / 16); v += kPPackThreads) {
        const int b = v / (kPWBytes / 16), x = v % (kPWBytes / 16);
        if (tile0 + b >= tiles) break;
        *reinterpret_cast<uint4 *>(out + ((tile0 + b) * nchunks + c) * kPBlockBytes + x * 16) =
            *reinterpret_cast<const uint4 *>(buf + (b * (kPWBytes / 16) + (x ^ (x >> 3 & 7))) * 4);
    }
    const int64_t g = k0 / group;
    for (int x = threadIdx.x; x < TILES * kPTileN; x += kPPackThreads) {
        const int64_t n = tile0 * kPTileN + x;
        if (tile0 + x / kPTileN >= tiles) break;
        T sv = from_float<T>(0.0f), tv = from_float<T>(0.0f);
        if (real && n < N) {
            sv = scale[g * N + n];
            if (offset != nullptr) tv = from_float<T>(to_float(offset[g * N + n]) * to_float(sv));
        }
        T *so = reinterpret_cast<T *>(out + ((tile0 + x / kPTileN) * nchunks + c) * kPBlockBytes + kPWBytes);
        so[x % kPTileN] = sv;
        so[kPTileN + x % kPTileN] = tv;
    }
}

// inverse of the weight part: one thread per stock word (k, i)
__global__ void __launch_bounds__(256)
w4a16_unpack_kernel(const uint8_t *__restrict__ packed, int64_t N, int64_t K, int nchunks, int32_t *__restrict__ w,
                    int64_t ld_w) {
    const int64_t words_n = N >> 3;
    const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= K * words_n) return;
    const int64_t k = idx / words_n, i = idx - k * words_n;
    const int c = static_cast<int>(k / kPChunkK), kc = static_cast<int>(k % kPChunkK);
    const int s = kc / kPSubK, kk = kc % kPSubK, e = kk & 7;
    const int pos = (e >> 1) + (e & 1) * 4;
    uint32_t word = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int64_t n = i * 8 + j;
        const int tile = static_cast<int>(n / kPTileN), r = static_cast<int>(n % kPTileN);
        const uint8_t *blk = packed + (static_cast<int64_t>(tile) * nchunks + c) * kPBlockBytes;
        const uint32_t pw = reinterpret_cast<const uint32_t *>(blk + (s * kPTileN + r) * 16)[kk >> 3];
        word |= ((pw >> (4 * pos)) & 15u) << (4 * j);
    }
    w[k * ld_w + i] = static_cast<int32_t>(word);
}

struct PPlan {
    int mpad, nblk, tiles_n, nchunks, grid, share, extra, grain, nstages, nxstages;
    size_t slots_bytes, smem;
};

PPlan p_make_plan(int64_t M, int64_t N, int64_t K) {
    PPlan pl;
    const int64_t sms = sm_count();
    pl.tiles_n = static_cast<int>((N + kPTileN - 1) / kPTileN);
    pl.nchunks = static_cast<int>((K + kPStageK - 1) / kPStageK);  // block pairs
    if (M <= kPMaxM) {
        pl.mpad = static_cast<int>((M + 15) / 16 * 16);
        pl.nblk = 1;
        pl.grain = 1;
        // activation tiles: enough to cover the L2 latency of their loads; the rest of the budget holds weights
        pl.nxstages = pl.mpad <= 16 ? 8 : (pl.mpad <= 32 ? 6 : 4);
        pl.nstages = static_cast<int>((kPSmemBudget - static_cast<size_t>(pl.nxstages) * pl.mpad * 512) / kPStageWBytes);
        if (pl.nstages > kPMaxStages) pl.nstages = kPMaxStages;
        pl.smem = 2048 + static_cast<size_t>(pl.nxstages) * pl.mpad * 512 + static_cast<size_t>(pl.nstages) * kPStageWBytes;
    } else {
        // Row tiles and the way of sharing them out by a model of the time (ns, fitted to 88 shapes of 65 .. 1500 rows, K of
        // 1024 .. 15232 and N of 1024 .. 28672, 4 to 20 plans each).  A stage takes what unpacking it takes (790) or its MMAs
        // (5 a row), a tile 61 a row more to leave tensor memory.  Whole tiles leave the last wave uneven; equal shares of the
        // stages do not, but every CTA then writes the sums of up to two tiles, and the one that arrives last at a tile adds
        // its slots one after the other: with few tiles that costs more than unpacking the weight again for lower row tiles
        // does (256 x 8192 x 1024: one row tile 42.0 us, four 14.9; 321 x 3584 x 1096: 18.8 / 11.7).  With many, as few row
        // tiles as the accumulator allows (1000 x 4096 x 28672: 201 us with four, 205 .. 226 with five to eight); a plan with
        // more has to be 6 % ahead.  The fit and these figures are older than the epilogue that loads one step ahead, which leaves
        // tensor memory in about half the time: where tiles are high and K is short the model is now above the measured
        // time (us, model / measured at the full clock: 1000 x 1024 x 28672 139 / 59, 1000 x 4096 x 28672 236 / 174,
        // 2048 x 4096 x 11008 184 / 140, 512 x 1024 x 8192 21 / 15).  With 30 for the 61, 6 % of the plans would differ; not measured.
        // A height of a multiple of 16 gives a number of row tiles, so there are sixteen candidates at most, whatever M is (a
        // search over the numbers took the host 31 us for 65536 rows, on each of a call's three visits here; 0.3 so).
        const int64_t fewest = (M + kPMaxWide - 1) / kPMaxWide;
        int64_t best = 0;
        for (int64_t mpad = kPMaxWide; mpad >= 16; mpad -= 16) {
            const int64_t nblk = (M + mpad - 1) / mpad;
            if (((M + nblk - 1) / nblk + 15) / 16 * 16 != mpad) continue;  // a lower tile gives as many
            if (nblk != fewest && nblk > M / 32) break;
            const int64_t tiles = pl.tiles_n * nblk, items = tiles * pl.nchunks, ctas = items < sms ? items : sms;
            const int64_t most = (items + ctas - 1) / ctas;
            const int64_t stage = 47 + mpad * 5 > 790 ? 47 + mpad * 5 : 790, drain = 61 * mpad;
            const int64_t whole = 99 + (tiles + sms - 1) / sms * (pl.nchunks * stage + drain);
            const int64_t slots = tiles < ctas ? 16 * ctas / tiles + 16 : 32;  // of a tile, in sixteenths
            const int64_t shared = 2187 + most * stage + drain * most / pl.nchunks + 35 * mpad + (mpad * 14 / 5 + 96) * slots / 16;
            const bool grain = whole <= shared || tiles > static_cast<int64_t>(kPCounterBytes / 4);  // (a counter a tile)
            const int64_t cost = (grain ? whole : shared) * (nblk == fewest ? 100 : 106);
            if (best == 0 || cost < best) {
                best = cost;
                pl.mpad = static_cast<int>(mpad);
                pl.nblk = static_cast<int>(nblk);
                pl.grain = grain ? pl.nchunks : 1;
            }
        }
        pl.nstages = kPWideStages;
        pl.nxstages = static_cast<int>((kPSmemBudgetWide - 2048 - kPWideStages * kPStageWBytes) / (static_cast<size_t>(pl.mpad) * 128));
        if (pl.nxstages > kPMaxXStages) pl.nxstages = kPMaxXStages;
        pl.smem = 2048 + static_cast<size_t>(pl.nxstages) * pl.mpad * 128 + static_cast<size_t>(pl.nstages) * kPStageWBytes;
        // more than half of an SM's: the next call's CTA is not placed beside this one, which holds all of the tensor memory (one of
        // the W8A8 cluster kernel with two an SM is, and waits for it)
        if (pl.smem < 120 * 1024) pl.smem = 120 * 1024;
    }
    const int64_t out_tiles = static_cast<int64_t>(pl.tiles_n) * pl.nblk;
    const int64_t grains = out_tiles * (pl.nchunks / pl.grain);
    pl.grid = static_cast<int>(grains < sms ? grains : sms);
    pl.share = static_cast<int>(grains / pl.grid);  // >= 1
    pl.extra = static_cast<int>(grains % pl.grid);
    // p_slot; none where no tile is shared: whole tiles, which a single block pair along K always is
    const int64_t slots = pl.grain == pl.nchunks ? 0 : pl.grid + (out_tiles < pl.grid ? out_tiles : pl.grid);
    pl.slots_bytes = static_cast<size_t>(slots) * pl.mpad * kPTileN * sizeof(float);
    return pl;
}

bool p_shape_ok(int64_t N, int64_t K, int64_t group) {
    return N > 0 && K > 0 && N % 8 == 0 && K % kPChunkK == 0 && group > 0 && group % kPChunkK == 0 && K % group == 0 &&
           K < (1ll << 31) && N < (1ll << 31) && (N + kPTileN - 1) / kPTileN <= static_cast<int64_t>(kPCounterBytes / 4);
}

// blocks along K, rounded up to an even count
int p_blocks_k(int64_t K) { return static_cast<int>((K + kPStageK - 1) / kPStageK) * kPPair; }

size_t p_packed_bytes(int64_t N, int64_t K) {
    return static_cast<size_t>((N + kPTileN - 1) / kPTileN) * static_cast<size_t>(p_blocks_k(K)) * kPBlockBytes;
}

// ---- one or two tokens of a large weight: integer dot products on the CUDA cores -------------------------
//
// The arithmetic of w4a16_gemv.cu (see there), which takes smaller weights.  Here the digits come from a small kernel in front
// and a thread reads its 64 bytes of a block straight from global memory (a warp's loads are 512 contiguous bytes); work is cut
// into equal contiguous runs of blocks, many CTAs per SM, and a tile's partial sums go to per-CTA slots that the last arriver
// adds in slot order, as in the tensor-core kernel.  Every further token adds 64 dp4a per block and thread, 7-8 us at 8192 x 28672,
// so beyond two tokens the tensor-core kernels are faster.  Measured slower: four columns per lane, which needs a quarter of the
// broadcast loads of digits (37 us against 33 us at two tokens); digits made by every CTA of 128 threads for its own blocks (30 us
// against 26 us); pulling lines of later blocks into L2 with prefetch instructions (29.6 us); mma.sync forms of the same idea
// (28 us at one token, 30 at eight, 42 at sixteen for int8 digits, 35 / 45 us with 16-bit operands, 43 / 71 us with e4m3, whose
// MMA is emulated).
constexpr int kGvMaxM = 2;            // measured (K=8192, N=28672): 26 / 33 us for 1 / 2 tokens, 41 / 51 us for 3 / 4
constexpr int kGvThreads = kPTileN;  // one output column per thread
constexpr int kGvCtasPerSm = 5;       // resident CTAs per SM (three blocks of weights in flight per thread; best of 4..8)

struct GvParams {
    const uint8_t *packed;
    const void *bias;
    void *out;
    int64_t ld_out;
    int N, tiles_n, nblocks, max_slots;
    int max_run;         // most blocks of one tile a CTA works on in a row (sizes the shared-memory copy of the digits)
    const uint4 *xd;     // digits [nblocks][M][2][8 x 16 bytes], bytes in the order the split words have
    const float *esc;    // [nblocks][M]
    const float *xs;     // [nblocks][M]
    float *slots;        // [tiles_n][max_slots][M][128]
    uint32_t *counters;  // [tiles_n], zero between calls
};

__device__ __forceinline__ uint4 ldg_stream(const uint8_t *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

template <typename T, int M>
__global__ void __launch_bounds__(kGvThreads, kGvCtasPerSm)
w4a16_gemv_kernel(GvParams p) {
    pdl_launch_dependents();
    extern __shared__ uint4 gv_smem[];  // digits of a run of blocks [nb][M][2][8], then esc [nb][M], xs [nb][M]
    __shared__ uint32_t s_is_last;
    const int r = threadIdx.x;
    const int64_t total = static_cast<int64_t>(p.tiles_n) * p.nblocks;
    const int64_t G = gridDim.x;
    const int64_t u_begin = total * blockIdx.x / G;
    const int64_t u_end = total * (blockIdx.x + 1) / G;
    const T *bias = static_cast<const T *>(p.bias);
    T *out = static_cast<T *>(p.out);
    bool waited = false;
    int64_t u = u_begin;
    while (u < u_end) {
        const int tile = static_cast<int>(u / p.nblocks);
        const int64_t tile_begin = static_cast<int64_t>(tile) * p.nblocks;
        const int64_t tile_end = tile_begin + p.nblocks;
        const int64_t seg_end = tile_end < u_end ? tile_end : u_end;
        const bool whole = (u == tile_begin && seg_end == tile_end);
        const int64_t n = static_cast<int64_t>(tile) * kPTileN + r;
        const bool n_ok = n < p.N;
        const int nb = static_cast<int>(seg_end - u), b_first = static_cast<int>(u - tile_begin);
        // the first two blocks' weights are on their way before anything else happens, the wait below included: see launch_pdl
        // for why that is safe
        const uint8_t *blk = p.packed + u * kPBlockBytes;
        uint4 wv[kPSubs], n1[kPSubs], n2[kPSubs];
#pragma unroll
        for (int s = 0; s < kPSubs; ++s) {
            wv[s] = ldg_stream(blk + (s * kPTileN + r) * 16);
            n1[s] = nb > 1 ? ldg_stream(blk + kPBlockBytes + (s * kPTileN + r) * 16) : make_uint4(0, 0, 0, 0);
        }
        T s_raw = *reinterpret_cast<const T *>(blk + kPWBytes + r * 2);
        T t_raw = *reinterpret_cast<const T *>(blk + kPWBytes + kPTileN * 2 + r * 2);
        // the digits come from the kernel launched just before this one (programmatic dependent launch: this
        // kernel may start while that one still runs)
        if (!waited) {
            pdl_wait();
            waited = true;
        }
        __syncthreads();  // the previous segment's digits are no longer read
        {
            const int nvec = nb * M * 16;
            const uint4 *src = p.xd + static_cast<int64_t>(b_first) * M * 16;
            for (int i = r; i < nvec; i += kGvThreads) gv_smem[i] = __ldg(src + i);
            float *tab = reinterpret_cast<float *>(gv_smem + p.max_run * M * 16);
            for (int i = r; i < nb * M; i += kGvThreads) {
                tab[i] = __ldg(p.esc + b_first * M + i);
                tab[p.max_run * M + i] = __ldg(p.xs + b_first * M + i);
            }
        }
        __syncthreads();
        const float *esc_s = reinterpret_cast<const float *>(gv_smem + p.max_run * M * 16);
        const float *xs_s = esc_s + p.max_run * M;
        float y[M];
#pragma unroll
        for (int m = 0; m < M; ++m) y[m] = 0.0f;
        for (int lb = 0; lb < nb; ++lb, blk += kPBlockBytes) {
            // the weights of the block after the next one are requested before this block is worked on
            if (lb + 2 < nb) {
#pragma unroll
                for (int s = 0; s < kPSubs; ++s) n2[s] = ldg_stream(blk + 2 * kPBlockBytes + (s * kPTileN + r) * 16);
            }
            T s_next = s_raw, t_next = t_raw;
            if (lb + 1 < nb) {
                s_next = *reinterpret_cast<const T *>(blk + kPBlockBytes + kPWBytes + r * 2);
                t_next = *reinterpret_cast<const T *>(blk + kPBlockBytes + kPWBytes + kPTileN * 2 + r * 2);
            }
            int d1[M], d2[M];
#pragma unroll
            for (int m = 0; m < M; ++m) d1[m] = d2[m] = 0;
            const uint4 *xd = gv_smem + lb * M * 16;
#pragma unroll
            for (int s = 0; s < kPSubs; ++s) {
                const uint32_t words[4] = {wv[s].x, wv[s].y, wv[s].z, wv[s].w};
#pragma unroll
                for (int h = 0; h < 2; ++h) {  // words 2h and 2h + 1 of the sub-step share one 16-byte digit vector
                    const uint32_t w0 = words[2 * h] ^ 0x88888888u, w1 = words[2 * h + 1] ^ 0x88888888u;
                    const int a0 = static_cast<int>(w0 & 0x0f0f0f0fu), b0 = static_cast<int>((w0 >> 4) & 0x0f0f0f0fu);
                    const int a1 = static_cast<int>(w1 & 0x0f0f0f0fu), b1 = static_cast<int>((w1 >> 4) & 0x0f0f0f0fu);
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const uint4 x1 = xd[(m * 2 + 0) * 8 + s * 2 + h];  // the same address in every lane: a broadcast
                        const uint4 x2 = xd[(m * 2 + 1) * 8 + s * 2 + h];
                        d1[m] = __dp4a(a0, static_cast<int>(x1.x), d1[m]);
                        d1[m] = __dp4a(b0, static_cast<int>(x1.y), d1[m]);
                        d1[m] = __dp4a(a1, static_cast<int>(x1.z), d1[m]);
                        d1[m] = __dp4a(b1, static_cast<int>(x1.w), d1[m]);
                        d2[m] = __dp4a(a0, static_cast<int>(x2.x), d2[m]);
                        d2[m] = __dp4a(b0, static_cast<int>(x2.y), d2[m]);
                        d2[m] = __dp4a(a1, static_cast<int>(x2.z), d2[m]);
                        d2[m] = __dp4a(b1, static_cast<int>(x2.w), d2[m]);
                    }
                }
            }
            const float sc = to_float(s_raw), tc = to_float(t_raw) - 8.0f * sc;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const float v = fmaf(static_cast<float>(d1[m]), 128.0f, static_cast<float>(d2[m]));
                y[m] = fmaf(sc * esc_s[lb * M + m], v, y[m]);
                y[m] = fmaf(tc, xs_s[lb * M + m], y[m]);
            }
#pragma unroll
            for (int s = 0; s < kPSubs; ++s) {
                wv[s] = n1[s];
                n1[s] = n2[s];
            }
            s_raw = s_next;
            t_raw = t_next;
        }
        const float bv = (n_ok && bias != nullptr) ? to_float(bias[n]) : 0.0f;
        if (whole) {
            if (n_ok) {
#pragma unroll
                for (int m = 0; m < M; ++m) out[static_cast<int64_t>(m) * p.ld_out + n] = from_float<T>(y[m] + bv);
            }
        } else {
            const int first_cta = p_cta_of_item(tile_begin, total, G);
            const int last_cta = p_cta_of_item(tile_end - 1, total, G);
            const int nslots = last_cta - first_cta + 1;
            const int64_t slot_elems = static_cast<int64_t>(M) * kPTileN;
            float *tile_slots = p.slots + static_cast<int64_t>(tile) * p.max_slots * slot_elems;
            float *mine = tile_slots + (static_cast<int>(blockIdx.x) - first_cta) * slot_elems + r;
#pragma unroll
            for (int m = 0; m < M; ++m) __stcg(mine + m * kPTileN, y[m]);
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) {
                const uint32_t old = atomicAdd(p.counters + tile, 1u);
                const bool is_last = (old + 1 == static_cast<uint32_t>(nslots));
                if (is_last) p.counters[tile] = 0;
                s_is_last = is_last ? 1u : 0u;
                __threadfence();
            }
            __syncthreads();
            if (s_is_last != 0 && n_ok) {
                float v[M];
#pragma unroll
                for (int m = 0; m < M; ++m) v[m] = 0.0f;
                for (int sl = 0; sl < nslots; ++sl) {
#pragma unroll
                    for (int m = 0; m < M; ++m) v[m] += __ldcg(tile_slots + sl * slot_elems + m * kPTileN + r);
                }
#pragma unroll
                for (int m = 0; m < M; ++m) out[static_cast<int64_t>(m) * p.ld_out + n] = from_float<T>(v[m] + bv);
            }
        }
        u = seg_end;
    }
}

// activations -> two int8 digits per element.  One warp per (block of 128 k, token): a lane takes four consecutive
// k (one 8-byte load), the block's absmax and sum are warp shuffles, no shared memory and no CTA barrier; the
// kernel is a few microseconds of latency in front of the matmul, so every step of it counts.
// grid (ceil(blocks / 4), M), 128 threads.
template <typename T>
__global__ void __launch_bounds__(128)
w4a16_gemv_digits_kernel(const T *__restrict__ x, int64_t ld_x, int M, int64_t K, int nblocks, int8_t *__restrict__ xd,
                         float *__restrict__ esc, float *__restrict__ xs) {
    pdl_wait();
    pdl_launch_dependents();  // not before the wait: the matmul reads its first weights without waiting for this kernel
    const int lane = threadIdx.x & 31;
    const int blk = blockIdx.x * 4 + (threadIdx.x >> 5), m = blockIdx.y;
    if (blk >= nblocks) return;
    const int64_t k0 = static_cast<int64_t>(blk) * kPChunkK + lane * 4;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (k0 < K) {  // K is a multiple of 128: a block is inside or a padding block
        const uint2 raw = __ldg(reinterpret_cast<const uint2 *>(x + static_cast<int64_t>(m) * ld_x + k0));
        const T *h = reinterpret_cast<const T *>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = to_float(h[j]);
    }
    float a = 0.0f;
    int bad = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float av = fabsf(v[j]);
        if (av <= 3.0e38f) a = fmaxf(a, av); else bad = 1;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    int e = 0, sum = 0;
    float e_scale = 0.0f;
    if (a > 0.0f) {
        (void)frexpf(a, &e);  // a = f * 2^e, f in [0.5, 1): |x| < 2^e; X = rint(x * 2^(14 - e))
        e_scale = ldexpf(1.0f, e - 14);
    }
    // byte positions inside the block's two 128-byte records (see the kernel's header for the order): the four k
    // of a lane lie in one group of eight, whose two words are bytes [8 g, 8 g + 8) of the sub-step's 32
    int8_t *rec = xd + (static_cast<int64_t>(blk) * M + m) * 256;
    const int s = lane >> 3, i = (lane >> 1) & 3;
    uint32_t d1w[2] = {0, 0}, d2w[2] = {0, 0};  // this lane's bytes of word A ([0]) and word B ([1]) of its group
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int X = 0;
        if (a > 0.0f) {
            float q = rintf(ldexpf(v[j], 14 - e));
            q = fminf(fmaxf(q, -16384.0f), 16383.0f);
            X = (q == q) ? static_cast<int>(q) : 0;
        }
        sum += X;
        const int e8 = (lane & 1) * 4 + j;                     // k within its group of eight
        const int pos = (e8 & 1) ? 4 + (e8 >> 1) : (e8 >> 1);  // nibble position of that k in the packed word
        const int word = pos & 1, byte = pos >> 1;
        d1w[word] |= (static_cast<uint32_t>(X >> 7) & 0xffu) << (8 * byte);
        d2w[word] |= (static_cast<uint32_t>(X & 127)) << (8 * byte);
    }
    // the two lanes of a group hold disjoint bytes of the same two words: merge them and let the even lane store
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        d1w[w] |= __shfl_xor_sync(0xffffffffu, d1w[w], 1);
        d2w[w] |= __shfl_xor_sync(0xffffffffu, d2w[w], 1);
    }
    if ((lane & 1) == 0) {
        *reinterpret_cast<uint2 *>(rec + s * 32 + i * 8) = make_uint2(d1w[0], d1w[1]);
        *reinterpret_cast<uint2 *>(rec + 128 + s * 32 + i * 8) = make_uint2(d2w[0], d2w[1]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) {
        // a block that holds a NaN or an infinity poisons the token's outputs, as the plain arithmetic would
        esc[blk * M + m] = bad ? __int_as_float(0x7fc00000) : e_scale;
        xs[blk * M + m] = e_scale * static_cast<float>(sum);  // |sum| < 2^21: exact
    }
}

struct GvPlan {
    int tiles_n, nblocks, grid, max_slots, max_run;
    size_t slots_bytes, xd_bytes, tab_bytes;
};

size_t gv_align256(size_t v) { return (v + 255) / 256 * 256; }

GvPlan gv_make_plan(int64_t M, int64_t N, int64_t K) {
    GvPlan pl;
    pl.tiles_n = static_cast<int>((N + kPTileN - 1) / kPTileN);
    pl.nblocks = p_blocks_k(K);
    const int64_t total = static_cast<int64_t>(pl.tiles_n) * pl.nblocks;
    const int64_t cap = static_cast<int64_t>(sm_count()) * kGvCtasPerSm;
    pl.grid = static_cast<int>(total < cap ? total : cap);
    const int64_t ipc = total / pl.grid;  // blocks per CTA, rounded down (>= 1)
    pl.max_slots = static_cast<int>((pl.nblocks + ipc - 1) / ipc + 1);
    pl.max_run = static_cast<int>(ipc + 1 < pl.nblocks ? ipc + 1 : pl.nblocks);
    pl.slots_bytes = gv_align256(static_cast<size_t>(pl.tiles_n) * pl.max_slots * M * kPTileN * sizeof(float));
    pl.xd_bytes = gv_align256(static_cast<size_t>(pl.nblocks) * M * 256);
    pl.tab_bytes = gv_align256(static_cast<size_t>(pl.nblocks) * M * sizeof(float));
    return pl;
}

size_t gv_workspace_bytes(int64_t M, int64_t N, int64_t K) {
    const GvPlan pl = gv_make_plan(M, N, K);
    return kPCounterBytes + pl.slots_bytes + pl.xd_bytes + 2 * pl.tab_bytes;
}

template <typename T>
int launch_gemv_t(const uint8_t *packed, const void *x, int64_t ld_x, const void *bias, void *out, int64_t ld_out,
                  int64_t M, int64_t N, int64_t K, void *workspace, cudaStream_t stream) {
    const GvPlan pl = gv_make_plan(M, N, K);
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    int8_t *xd = reinterpret_cast<int8_t *>(ws + kPCounterBytes + pl.slots_bytes);
    float *esc = reinterpret_cast<float *>(ws + kPCounterBytes + pl.slots_bytes + pl.xd_bytes);
    float *xs = reinterpret_cast<float *>(ws + kPCounterBytes + pl.slots_bytes + pl.xd_bytes + pl.tab_bytes);
    QMM_CUDA_OK(launch_pdl(w4a16_gemv_digits_kernel<T>, dim3(static_cast<unsigned>((pl.nblocks + 3) / 4), static_cast<unsigned>(M)),
                           dim3(128), 0, stream, static_cast<const T *>(x), ld_x, static_cast<int>(M), K, pl.nblocks, xd, esc, xs));
    GvParams p;
    p.packed = packed;
    p.bias = bias;
    p.out = out;
    p.ld_out = ld_out;
    p.N = static_cast<int>(N);
    p.tiles_n = pl.tiles_n;
    p.nblocks = pl.nblocks;
    p.max_slots = pl.max_slots;
    p.max_run = pl.max_run;
    p.xd = reinterpret_cast<const uint4 *>(xd);
    p.esc = esc;
    p.xs = xs;
    p.counters = reinterpret_cast<uint32_t *>(ws);
    p.slots = reinterpret_cast<float *>(ws + kPCounterBytes);
    // programmatic dependent launch: the kernel starts (and requests its first weights) while the digits
    // kernel still runs, and waits for it (griddepcontrol.wait) before it reads the digits
    const size_t smem = static_cast<size_t>(pl.max_run) * M * (256 + 8);
    auto launch = [&](auto kern) -> int {
        if (smem > 48 * 1024)
            QMM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        QMM_CUDA_OK(launch_pdl(kern, dim3(static_cast<unsigned>(pl.grid)), dim3(kGvThreads), smem, stream, p));
        return QMM_OK;
    };
    switch (M) {
        case 1: return launch(w4a16_gemv_kernel<T, 1>);
        default: return launch(w4a16_gemv_kernel<T, 2>);  // kGvMaxM
    }
}

template <typename T>
int launch_prepacked_t(const uint8_t *packed, const void *x, int64_t ld_x, const void *bias, void *out, int64_t ld_out,
                       int64_t M, int64_t N, int64_t K, const BTables *tables, void *workspace, cudaStream_t stream) {
    const PPlan pl = p_make_plan(M, N, K);
    PParams p;
    p.packed = packed;
    p.bias = bias;
    p.out = out;
    p.ld_out = ld_out;
    p.M = static_cast<int>(M);
    p.N = static_cast<int>(N);
    p.mpad = pl.mpad;
    p.nblk = pl.nblk;
    p.share = pl.share;
    p.extra = pl.extra;
    p.grain = pl.grain;
    p.out_vec = (reinterpret_cast<uintptr_t>(out) & 7) == 0 && (ld_out & 3) == 0;
    p.x_box_bytes = pl.mpad * 128;
    p.nstages = pl.nstages;
    p.nxstages = pl.nxstages;
    p.tiles_n = pl.tiles_n;
    p.nchunks = pl.nchunks;
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    p.counters = reinterpret_cast<uint32_t *>(ws);
    p.slots = reinterpret_cast<float *>(ws + kPCounterBytes);
    p.status = device_status_word();

    CUtensorMap tx;
    int rc = make_tmap_2d(&tx, x, 2, static_cast<uint64_t>(K), static_cast<uint64_t>(M), static_cast<uint64_t>(ld_x), 64,
                          static_cast<uint32_t>(pl.mpad), true);
    if (rc != QMM_OK) return rc;
    static_assert(sizeof(PSmemTail) <= 1024 && sizeof(BSmemTail) <= 1024, "the tail has 1 KiB");
    if (tables != nullptr && M <= kBTok) {
        auto kern = w4a16_block_kernel<T>;
        QMM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(pl.smem)));
        QMM_CUDA_OK(launch_pdl(kern, dim3(static_cast<unsigned>(pl.grid)), dim3(kPThreads), pl.smem, stream, tx, p, *tables));
        return QMM_OK;
    }
    auto kern = M <= kPMaxM ? w4a16_prepacked_kernel<T, false> : w4a16_prepacked_kernel<T, true>;
    QMM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(pl.smem)));
    QMM_CUDA_OK(launch_pdl(kern, dim3(static_cast<unsigned>(pl.grid)), dim3(kPThreads), pl.smem, stream, tx, p));
    return QMM_OK;
}

}  // namespace
}  // namespace qmm

extern "C" int qmm_w4a16_prepack_size(int64_t N, int64_t K, int64_t group, size_t *bytes) {
    using namespace qmm;
    QMM_REQUIRE(bytes != nullptr, "qmm_w4a16_prepack_size: bytes is NULL");
    *bytes = p_shape_ok(N, K, group > 0 ? group : K) ? p_packed_bytes(N, K) : 0;
    return QMM_OK;
}

extern "C" int qmm_w4a16_prepack(const int32_t *weight, int64_t ld_w, const void *antiquant_scale,
                                 const void *antiquant_offset, int sdtype, int64_t group, int64_t N, int64_t K,
                                 void *packed, size_t packed_bytes, void *stream) {
    using namespace qmm;
    if (group <= 0) group = K;
    QMM_REQUIRE(sdtype == QMM_DTYPE_BF16 || sdtype == QMM_DTYPE_F16, "qmm_w4a16_prepack: scale must be bf16 or f16");
    if (!p_shape_ok(N, K, group))
        return fail(QMM_ERR_UNSUPPORTED,
                    "qmm_w4a16_prepack: needs N % 8 == 0, K % 128 == 0 and a group that is a multiple of 128 dividing K");
    QMM_REQUIRE(weight != nullptr && antiquant_scale != nullptr && packed != nullptr, "qmm_w4a16_prepack: NULL operand");
    QMM_REQUIRE(ld_w >= N / 8, "qmm_w4a16_prepack: ld_w smaller than N/8");
    QMM_REQUIRE((reinterpret_cast<uintptr_t>(packed) & 15) == 0, "qmm_w4a16_prepack: packed must be 16-byte aligned");
    if (packed_bytes < p_packed_bytes(N, K))
        return fail(QMM_ERR_WORKSPACE, "qmm_w4a16_prepack: packed buffer smaller than qmm_w4a16_prepack_size");
    const int nchunks = p_blocks_k(K);
    const int64_t tiles = (N + kPTileN - 1) / kPTileN;
    QMM_REQUIRE(tiles <= 65535, "qmm_w4a16_prepack: N too large");
    const int aligned = (reinterpret_cast<uintptr_t>(weight) & 15) == 0 && (ld_w & 3) == 0;
    const int per_cta = (tiles + 3) / 4 * nchunks >= sm_count() ? 4 : 1;
    const dim3 grid(static_cast<unsigned>(nchunks), static_cast<unsigned>((tiles + per_cta - 1) / per_cta));
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto launch = [&](auto kern, auto type) {
        using T = decltype(type);
        return launch_pdl(kern, grid, dim3(kPPackThreads), 0, s, weight, ld_w, aligned, static_cast<const T *>(antiquant_scale),
                          static_cast<const T *>(antiquant_offset), group, N, K, nchunks, static_cast<uint8_t *>(packed));
    };
    if (sdtype == QMM_DTYPE_BF16)
        QMM_CUDA_OK(launch(per_cta == 1 ? w4a16_prepack_kernel<__nv_bfloat16, 1> : w4a16_prepack_kernel<__nv_bfloat16, 4>,
                           __nv_bfloat16()));
    else
        QMM_CUDA_OK(launch(per_cta == 1 ? w4a16_prepack_kernel<__half, 1> : w4a16_prepack_kernel<__half, 4>, __half()));
    return QMM_OK;
}

extern "C" int qmm_w4a16_unpack_weight(const void *packed, int64_t N, int64_t K, int32_t *weight, int64_t ld_w,
                                       void *stream) {
    using namespace qmm;
    if (!p_shape_ok(N, K, K)) return fail(QMM_ERR_UNSUPPORTED, "qmm_w4a16_unpack_weight: needs N % 8 == 0 and K % 128 == 0");
    QMM_REQUIRE(packed != nullptr && weight != nullptr, "qmm_w4a16_unpack_weight: NULL operand");
    QMM_REQUIRE(ld_w >= N / 8, "qmm_w4a16_unpack_weight: ld_w smaller than N/8");
    const int64_t total = K * (N / 8);
    w4a16_unpack_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t *>(packed), N, K, p_blocks_k(K), weight, ld_w);
    QMM_CUDA_OK(cudaGetLastError());
    return QMM_OK;
}

extern "C" int qmm_weight_quant_batchmatmul_prepacked_workspace_size(int64_t M, int64_t N, int64_t K, size_t *bytes) {
    using namespace qmm;
    QMM_REQUIRE(bytes != nullptr, "qmm_weight_quant_batchmatmul_prepacked_workspace_size: bytes is NULL");
    QMM_REQUIRE(M >= 0 && N >= 0 && K >= 0, "qmm_weight_quant_batchmatmul_prepacked_workspace_size: negative argument");
    *bytes = 0;
    if (M > 0 && p_shape_ok(N, K, K)) {
        *bytes = kPCounterBytes + p_make_plan(M, N, K).slots_bytes;
        if (M <= kGvMaxM && gv_workspace_bytes(M, N, K) > *bytes) *bytes = gv_workspace_bytes(M, N, K);
    }
    return QMM_OK;
}

namespace qmm {
namespace {
int prepacked_matmul(const void *x, int x_dtype, int64_t ld_x, const void *packed, size_t packed_bytes, const BTables *tables,
                     const void *bias, void *out, int64_t ld_out, int64_t M, int64_t N, int64_t K, void *workspace,
                     size_t workspace_bytes, void *stream) {
    QMM_REQUIRE(M >= 0, "qmm_weight_quant_batchmatmul_prepacked: negative M");
    QMM_REQUIRE(x_dtype == QMM_DTYPE_BF16 || x_dtype == QMM_DTYPE_F16,
                "qmm_weight_quant_batchmatmul_prepacked: x must be bf16 or f16");
    if (!p_shape_ok(N, K, K))
        return fail(QMM_ERR_UNSUPPORTED, "qmm_weight_quant_batchmatmul_prepacked: needs N % 8 == 0 and K % 128 == 0");
    if (M == 0) return QMM_OK;
    QMM_REQUIRE(x != nullptr && packed != nullptr && out != nullptr, "qmm_weight_quant_batchmatmul_prepacked: NULL operand");
    QMM_REQUIRE(ld_x >= K && ld_out >= N, "qmm_weight_quant_batchmatmul_prepacked: row pitch smaller than the row");
    QMM_REQUIRE(packed_bytes >= p_packed_bytes(N, K),
                "qmm_weight_quant_batchmatmul_prepacked: packed buffer smaller than qmm_w4a16_prepack_size");
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (ld_x & 7) || (reinterpret_cast<uintptr_t>(packed) & 15))
        return fail(QMM_ERR_UNSUPPORTED,
                    "qmm_weight_quant_batchmatmul_prepacked: x and packed need 16-byte aligned addresses and row pitch");
    size_t need = 0;
    qmm_weight_quant_batchmatmul_prepacked_workspace_size(M, N, K, &need);
    if (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 255) != 0 || workspace_bytes < need)
        return fail(QMM_ERR_WORKSPACE,
                    "qmm_weight_quant_batchmatmul_prepacked: workspace missing, not 256-byte aligned or too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (prefer_gemv_tile(M, N, K)) return launch_gemv_tile(packed, x, x_dtype, ld_x, bias, out, ld_out, M, N, K, s);
    if (M <= kGvMaxM)  // a handful of tokens: dp4a on the CUDA cores, at the speed of the weight stream
        return (x_dtype == QMM_DTYPE_BF16)
                   ? launch_gemv_t<__nv_bfloat16>(static_cast<const uint8_t *>(packed), x, ld_x, bias, out, ld_out, M, N, K,
                                                  workspace, s)
                   : launch_gemv_t<__half>(static_cast<const uint8_t *>(packed), x, ld_x, bias, out, ld_out, M, N, K,
                                           workspace, s);
    return (x_dtype == QMM_DTYPE_BF16)
               ? launch_prepacked_t<__nv_bfloat16>(static_cast<const uint8_t *>(packed), x, ld_x, bias, out, ld_out, M, N, K,
                                                   tables, workspace, s)
               : launch_prepacked_t<__half>(static_cast<const uint8_t *>(packed), x, ld_x, bias, out, ld_out, M, N, K,
                                            tables, workspace, s);
}
}  // namespace
}  // namespace qmm

extern "C" int qmm_weight_quant_batchmatmul_prepacked(const void *x, int x_dtype, int64_t ld_x, const void *packed,
                                                      size_t packed_bytes, const void *bias, void *out,
                                                      int64_t ld_out, int64_t M, int64_t N, int64_t K,
                                                      void *workspace, size_t workspace_bytes, void *stream) {
    return qmm::prepacked_matmul(x, x_dtype, ld_x, packed, packed_bytes, nullptr, bias, out, ld_out, M, N, K, workspace,
                                 workspace_bytes, stream);
}

extern "C" int qmm_weight_quant_batchmatmul_prepacked_tables(const void *x, int x_dtype, int64_t ld_x, const void *packed,
                                                             size_t packed_bytes, const void *antiquant_scale,
                                                             const void *antiquant_offset, int64_t group, const void *bias,
                                                             void *out, int64_t ld_out, int64_t M, int64_t N, int64_t K,
                                                             void *workspace, size_t workspace_bytes, void *stream) {
    using namespace qmm;
    if (group <= 0) group = K;
    if (!p_shape_ok(N, K, group))
        return fail(QMM_ERR_UNSUPPORTED, "qmm_weight_quant_batchmatmul_prepacked_tables: needs N % 8 == 0, K % 128 == 0 and a "
                                         "group that is a multiple of 128 dividing K");
    QMM_REQUIRE(antiquant_scale != nullptr, "qmm_weight_quant_batchmatmul_prepacked_tables: NULL scale");
    BTables t;
    t.scale = antiquant_scale;
    t.offset = antiquant_offset;
    t.group_blocks = static_cast<int>(group / kPChunkK);
    t.nblocks = static_cast<int>(K / kPChunkK);
    t.x = x;
    t.ld_x = ld_x;
    // the tables' rows are fetched by copies of whole 16 bytes
    const bool aligned = ((reinterpret_cast<uintptr_t>(antiquant_scale) | reinterpret_cast<uintptr_t>(antiquant_offset)) & 15) == 0;
    return prepacked_matmul(x, x_dtype, ld_x, packed, packed_bytes, aligned ? &t : nullptr, bias, out, ld_out, M, N, K, workspace,
                            workspace_bytes, stream);
}
