// W8A8 matmul for shapes whose output tiles do not fill the GPU: K is cut over the CTA pairs of a cluster.
//
// One cluster works on one output tile of 256 columns x T tokens (T = 32 .. 256 in steps of 32).  The weights are the MMA's M
// operand, so a token tile is as high as the call needs and not 128 or 256 rows.  A pair of CTAs runs
// tcgen05.mma.cta_group::2 (256 x T x 32) on its slice of K: each CTA loads 128 weight columns and half of the tokens.  With
// S = 2 or 4 slices the cluster holds S pairs, whose int32 sums meet in shared memory: CTA (slice s, half r) owns the
// tokens [s T / S, (s + 1) T / S) of its 128 columns, receives the other slices' sums for them through distributed shared
// memory and finishes them.  No scratch in global memory, no atomics, no second launch, and integer sums: the result does
// not depend on how K is cut.
//
// A thread of the epilogue owns a column.  Its scale and bias are loaded while the main loop runs, as are the tokens' scales:
// with one tile a CTA nothing else hides those loads (the tile kernel fetches them for every 64 columns, between two loads
// from tensor memory).
//
// What bounds it and what it measured (us, M x K x N, bf16, the kernel replayed in a CUDA graph, operands rotated past L2; this / the best
// of the tile, split-K, stream-K and CTA-pair kernels; a call through the operator takes up to 1 us more).  Small: launch, first data and the
// hand-offs: 128 x 1024 x 1024 3.9 / 7.5, 64 x 1024 x 8192 4.7 / 7.8 (stream-K, which used to take it, 38.7), 1 x 4096 x 4096 7.2 / 12.1.
// Decode: HBM: 1 x 8192 x 28672 39.2 / 46.2 (36.4 at the copy rate), 32 x 28672 x 8192 38.9 / 46.1 (36.6).  A prompt of some hundred tokens:
// shared memory's fill from L2, about 105 B/ns an SM, then the MMA rate: 333 x 4096 x 6144 11.3 / 16.5, 512 x 14336 x 4096 25.9 / 38.3.
//
// Synchronisation of a pair (s = stage): full[s] on the pair's leader counts the bytes of both CTAs' loads; empty[s] and done,
// one per CTA, are arrived on by the leader's tcgen05.commit.  Cluster barriers separate the end of all main loops (the
// operand rings become receive buffers), the exchange, and the exit.  No TMA load uses multicast; every wait is bounded.
#include <algorithm>
#include <type_traits>

#include "qmm_common.cuh"
#include "w8a8_epilogue.cuh"

namespace qmm {

namespace {

constexpr int kCUnitN = 256;   // columns of a pair's tile
constexpr int kCBK = 128;      // k elements per stage
constexpr int kCWBytes = (kCUnitN / 2) * kCBK;  // weights of a stage and CTA
constexpr int kCMaxT = 256;
constexpr int kCMaxStages = 8;
constexpr int kCEpiWarps = 8;  // two for each quarter of the tensor memory lanes (16: 0.3 us more at 128 x 1024 x 1024)
constexpr int kCParts = kCEpiWarps / 4;
constexpr int kCThreads = (2 + kCEpiWarps) * 32;
constexpr int kCMaxSmem = 220 * 1024;

struct ClusterSmemTail {
    uint64_t full[kCMaxStages];
    uint64_t empty[kCMaxStages];
    uint64_t done;
    uint32_t tmem_base;
    uint32_t abort_flag;
    float pertoken[kCMaxT];
};

struct ClusterParams {
    EpilogueParams ep;
    int num_kb;
    int T;            // tokens of a tile, a multiple of 32
    int tiles_m;      // token tiles
    int stages;
    int stage_bytes;  // kCWBytes + T / 2 * kCBK
    uint32_t tmem_cols;
    uint32_t *status;
};

__device__ __forceinline__ void cluster_epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kCEpiWarps * 32) : "memory"); }

// 32 lanes x 8 consecutive 32-bit columns; complete after tmem_ld_wait()
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

template <typename OutT, bool W_MN_MAJOR, int S>
__global__ void __launch_bounds__(kCThreads, 2)
w8a8_cluster_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, ClusterParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t smem_base = smem_u32(smem_raw);
    ClusterSmemTail *tail = reinterpret_cast<ClusterSmemTail *>(smem_raw + p.stages * p.stage_bytes);
    volatile uint32_t *abort_flag = &tail->abort_flag;
    // the CTAs of a cluster see the same alignment, so this exit is taken by all or by none
    if ((smem_base & 1023u) != 0) {
        if (threadIdx.x == 0 && p.status != nullptr) atomicMax(p.status, DEV_STATUS_SMEM_MISALIGNED);
        return;
    }
    const int warp = warp_id_uniform();
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int half = static_cast<int>(rank & 1);      // columns [128 half, +128) of the tile, tokens [T / 2 half, +T / 2)
    const int slice = static_cast<int>(rank >> 1);
    const uint32_t leader_rank = rank & ~1u;
    const bool leader = half == 0;
    // token tiles run fastest: those of the same columns find the weights in L2
    const int tile = static_cast<int>(blockIdx.x / (2 * S));
    const int n0 = tile / p.tiles_m * kCUnitN, m0 = tile % p.tiles_m * p.T;
    const int kb_begin = static_cast<int>(static_cast<int64_t>(p.num_kb) * slice / S);
    const int kb_end = static_cast<int>(static_cast<int64_t>(p.num_kb) * (slice + 1) / S);

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&tail->full[s]), 1);
            mbar_init(smem_u32(&tail->empty[s]), 1);
        }
        mbar_init(smem_u32(&tail->done), 1);
        tail->abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmap_w);
        tma_prefetch_desc(&tmap_x);
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(&tail->tmem_base), p.tmem_cols);
        tmem_relinquish_pair();
        pdl_launch_dependents();
    }
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the peer's barriers are initialised before anything signals them
    tc_fence_after();
    const uint32_t tmem_base = warp_uniform(tail->tmem_base);

    const EpilogueParams &ep = p.ep;
    const int quarter = warp & 3, part = (warp - 2) >> 2;  // epilogue warps: lanes, and which groups of eight tokens
    const int col = quarter * 32 + lane;
    const int n = n0 + half * (kCUnitN / 2) + col;
    const int own = p.T / S;               // tokens that this CTA finishes
    const int own0 = slice * own;          // first of them within the tile
    constexpr bool is_i8 = sizeof(OutT) == 1, is_i32 = sizeof(OutT) == 4;
    const bool has_pt = !is_i32 && ep.pertoken_scale != nullptr;
    const bool has_add = is_i8 ? ep.offset != nullptr
                               : !is_i32 && ep.bias != nullptr && ep.bias_dtype != QMM_DTYPE_NONE && ep.bias_dtype != QMM_DTYPE_I32;
    float scale = 0.0f, add = 0.0f;  // add: the bias of a 16-bit output, the offset of an int8 one
    int32_t ibias = 0;               // of an int32 or int8 output
    bool ok = true;

    if (warp == 0) {
        // ---------------- TMA producer (every CTA) ----------------
        uint32_t stage = 0, phase = 0;
        for (int kb = kb_begin; kb < kb_end; ++kb) {
            if (!mbar_wait(smem_u32(&tail->empty[stage]), phase ^ 1, abort_flag, 0x61)) break;
            if (lane == 0) {
                const uint32_t full_local = smem_u32(&tail->full[stage]);
                const uint32_t full_leader = map_to_cta(full_local, leader_rank);
                const uint32_t sw = smem_base + stage * p.stage_bytes;
                if (leader) mbar_expect_tx(full_local, 2 * p.stage_bytes);
                if (W_MN_MAJOR)
                    tma_load_2d_pair(sw, &tmap_w, n0 + half * (kCUnitN / 2), kb * kCBK, full_leader);  // [128 k-rows][128 n-bytes]
                else
                    tma_load_2d_pair(sw, &tmap_w, kb * kCBK, n0 + half * (kCUnitN / 2), full_leader);  // [128 n-rows][128 k-bytes]
                tma_load_2d_pair(sw + kCWBytes, &tmap_x, kb * kCBK, m0 + half * (p.T / 2), full_leader);  // [T/2 tokens][128 k-bytes]
            }
            __syncwarp();
            if (++stage == static_cast<uint32_t>(p.stages)) {
                stage = 0;
                phase ^= 1;
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader of each pair) ----------------
        if (leader) {
            const uint32_t idesc = make_idesc(/*c=s32*/ 2, 1, 1, W_MN_MAJOR ? 1u : 0u, /*b K-major*/ 0, kCUnitN,
                                              static_cast<uint32_t>(p.T));
            constexpr uint32_t kDescHi = smem_desc_hi_sw128(1024);
            constexpr uint32_t kAStep = W_MN_MAJOR ? (4096u >> 4) : 2u;  // per 32-element K step
            const uint32_t a_lo0 = smem_desc_lo(smem_base, W_MN_MAJOR ? 1024u : 16u);
            const uint32_t b_lo0 = smem_desc_lo(smem_base + kCWBytes, 16);
            const uint32_t stage_step = static_cast<uint32_t>(p.stage_bytes) >> 4;
            const uint32_t full0 = smem_u32(&tail->full[0]), empty0 = smem_u32(&tail->empty[0]);
            const uint16_t mask = static_cast<uint16_t>(0x3u << leader_rank);
            uint32_t stage = 0, phase = 0, accumulate = 0;
            for (int kb = kb_begin; kb < kb_end; ++kb) {
                ok = mbar_wait(full0 + stage * 8, phase, abort_flag, 0x62);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a_lo = a_lo0 + stage * stage_step, b_lo = b_lo0 + stage * stage_step;
#pragma unroll
                for (int k = 0; k < kCBK / 32; ++k) {
                    mma_i8_ss_pair_warp(tmem_base, desc64(a_lo + kAStep * k, kDescHi), desc64(b_lo + 2 * k, kDescHi), idesc,
                                        accumulate);
                    accumulate = 1;
                }
                tc_commit_pair_warp(empty0 + stage * 8, mask);
                if (++stage == static_cast<uint32_t>(p.stages)) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            if (ok) tc_commit_pair_warp(smem_u32(&tail->done), mask);
        }
    } else {
        // ---------------- epilogue warps: constants, then wait for the sums ----------------
        if (n < ep.N) {
            if constexpr (!is_i32) {
                scale = ep.scale_is_scalar ? __ldg(ep.scale) : __ldg(ep.scale + n);
                if (has_add) {
                    if constexpr (is_i8)
                        add = ep.offset_is_scalar ? __ldg(ep.offset) : __ldg(ep.offset + n);
                    else
                        add = load_bias_f32(ep, n);
                }
            }
            if constexpr (is_i8 || is_i32) {
                if (ep.bias != nullptr && ep.bias_dtype == QMM_DTYPE_I32) ibias = __ldg(static_cast<const int32_t *>(ep.bias) + n);
            }
        }
        for (int t = threadIdx.x - 64; t < own; t += kCEpiWarps * 32) {
            const int m = m0 + own0 + t;
            tail->pertoken[t] = has_pt && m < ep.M ? __ldg(ep.pertoken_scale + m) : 1.0f;
        }
        cluster_epi_sync();
        ok = mbar_wait(smem_u32(&tail->done), 0, abort_flag, 0x63);
        tc_fence_after();
    }
    __syncwarp();

    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    // sums of the other slices for this CTA's tokens: [source][group of four tokens][128 columns] x 16 bytes, over the ring
    const int groups = own / 8;
    if constexpr (S > 1) {
        cluster_sync_all();  // every pair's MMAs are complete: nothing reads or fills a ring any more
        if (warp >= 2 && ok) {
            // four groups' loads from tensor memory under way at a time
            for (int i0 = part; i0 < (S - 1) * groups; i0 += 4 * kCParts) {
                uint32_t v[4][8];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int i = i0 + kCParts * b, d = i / groups;
                    if (i < (S - 1) * groups) tmem_ld_32x8(taddr + (d + (d >= slice ? 1 : 0)) * own + (i - d * groups) * 8, v[b]);
                }
                tmem_ld_wait();
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int i = i0 + kCParts * b, d = i / groups, g = i - d * groups, dst = d + (d >= slice ? 1 : 0);
                    if (i >= (S - 1) * groups) break;
                    const int src = slice < dst ? slice : slice - 1;
                    const uint32_t at = map_to_cta(smem_base + ((src * groups + g) * 2 * 128 + col) * 16, static_cast<uint32_t>(dst * 2 + half));
                    st_cluster_v4(at, v[b][0], v[b][1], v[b][2], v[b][3]);
                    st_cluster_v4(at + 128 * 16, v[b][4], v[b][5], v[b][6], v[b][7]);
                }
            }
        }
        cluster_sync_all();  // the sums have arrived
    }
    if (warp >= 2 && ok) {
        OutT *out = static_cast<OutT *>(ep.out) + n;
        const int4 *recv = reinterpret_cast<const int4 *>(smem_raw) + col;
        const bool pairs_ok = (reinterpret_cast<uintptr_t>(ep.out) & (2 * sizeof(OutT) - 1)) == 0 && (ep.ld_out & 1) == 0;
        for (int g0 = part; g0 < groups; g0 += 2 * kCParts) {
            uint32_t v[2][8];
#pragma unroll
            for (int b = 0; b < 2; ++b)
                if (g0 + kCParts * b < groups) tmem_ld_32x8(taddr + own0 + (g0 + kCParts * b) * 8, v[b]);
            tmem_ld_wait();
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int g = g0 + kCParts * b, m = m0 + own0 + g * 8;
                if (g >= groups || m >= ep.M) break;
                int32_t acc[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = static_cast<int32_t>(v[b][j]);
                if constexpr (S > 1) {
#pragma unroll
                    for (int s = 0; s < S - 1; ++s) {
                        const int4 r0 = recv[(s * groups + g) * 2 * 128], r1 = recv[((s * groups + g) * 2 + 1) * 128];
                        acc[0] += r0.x, acc[1] += r0.y, acc[2] += r0.z, acc[3] += r0.w;
                        acc[4] += r1.x, acc[5] += r1.y, acc[6] += r1.z, acc[7] += r1.w;
                    }
                }
                const float4 p0 = *reinterpret_cast<const float4 *>(tail->pertoken + g * 8), p1 = *reinterpret_cast<const float4 *>(tail->pertoken + g * 8 + 4);
                const float pt[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
                if constexpr (is_i32) {
                    if (n >= ep.N) continue;
                    OutT *o = out + static_cast<int64_t>(m) * ep.ld_out;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (m + j < ep.M) o[j * ep.ld_out] = acc[j] + ibias;
                } else {
                    // two lanes swap halves: each then stores two neighbouring columns of four tokens
                    uint32_t lo[2], hi[2];  // column n & ~1 and the next one; four tokens, two (16-bit) or four (int8) a word
                    constexpr int kWords = is_i8 ? 1 : 2;
#pragma unroll
                    for (int i = 0; i < kWords; ++i) {
                        uint32_t first, second;  // this column's tokens of the even lane, and of the odd one
                        if constexpr (is_i8) {
                            first = second = 0;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                first |= (requant_one(acc[j] + ibias, scale, pt[j], has_pt, add, has_add) & 0xffu) << (8 * j);
                                second |= (requant_one(acc[4 + j] + ibias, scale, pt[4 + j], has_pt, add, has_add) & 0xffu) << (8 * j);
                            }
                        } else {
                            auto value = [&](int j) { return dequant_one(acc[j], scale, pt[j], has_pt, add, has_add); };
                            first = pack2<OutT>(value(2 * i), value(2 * i + 1));
                            second = pack2<OutT>(value(4 + 2 * i), value(4 + 2 * i + 1));
                        }
                        const bool odd = lane & 1;
                        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? first : second, 1);
                        lo[i] = odd ? got : first;
                        hi[i] = odd ? second : got;
                    }
                    const int mt = m + (lane & 1) * 4;
                    OutT *o = out - (lane & 1) + static_cast<int64_t>(mt) * ep.ld_out;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (mt + j >= ep.M) break;
                        OutT *at = o + j * ep.ld_out;
                        // the pair's bytes: of token j
                        const uint32_t two = is_i8 ? __byte_perm(lo[0], hi[0], j | (4 + j) << 4)
                                                   : __byte_perm(lo[j >> (is_i8 ? 8 : 1)], hi[j >> (is_i8 ? 8 : 1)], j & 1 ? 0x7632 : 0x5410);
                        using Pair = typename std::conditional<is_i8, uint16_t, uint32_t>::type;
                        using One = typename std::conditional<is_i8, uint8_t, uint16_t>::type;
                        if (pairs_ok && (n | 1) < ep.N) {
                            *reinterpret_cast<Pair *>(at) = static_cast<Pair>(two);
                        } else {
                            if ((n & ~1) < ep.N) *reinterpret_cast<One *>(at) = static_cast<One>(two);
                            if ((n | 1) < ep.N) *reinterpret_cast<One *>(at + 1) = static_cast<One>(two >> (8 * sizeof(OutT)));
                        }
                    }
                }
            }
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && tail->abort_flag != 0 && p.status != nullptr) atomicMax(p.status, tail->abort_flag);
    cluster_sync_all();  // nobody signals a CTA that already left; both CTAs of a pair are done with their tensor memory
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, p.tmem_cols);
    }
}

struct ClusterPlan {
    int T = 0, slices = 0, stages = 0, stage_bytes = 0;
    int64_t clusters = 0;
    size_t smem = 0;
    uint32_t tmem_cols = 32;
};

// Stages of the operand ring.  Two CTAs of an SM never want more tensor memory (T <= 256 columns each) or shared memory than it
// has; three do not fit.
int cluster_stages(int stage_bytes, bool two) {
    const int budget = (two ? kCMaxSmem / 2 : kCMaxSmem) - static_cast<int>(sizeof(ClusterSmemTail));
    return std::min(kCMaxStages, budget / stage_bytes);
}

// Token height and number of K slices by a model of the time (ns, fitted to about 190 shapes of 1 .. 2048 tokens, K and N of
// 1024 .. 28672, every T and S each; its choice takes 0.5 % more than the best one on average, 10 % at most):
//   a k block of a CTA takes what its loads take at 105 B/ns or what its MMAs take, 1.4 ns a token;
//   the CTAs of all SMs together load 14 B/ps;  memory delivers what the call cannot do without at 6.5 B/ps;
//   the exchange of two slices takes 1.2 us, of four 2.4 us, and 12 ns a token.
// Only plans whose clusters are all resident at once: one CTA an SM with a deep ring, or two with half of it each where the
// clusters are more than that.  (Beyond, the persistent CTA-pair kernel is ahead: 700 x 4096 x 28672 73 us here, 66 there.)
// `resident`: clusters of S = 1, 2, 4 slices that fit with one CTA an SM, as cudaOccupancyMaxActiveClusters says for 148 SMs;
// the SMs of a GPC that do not fill a cluster stay idle.
bool cluster_make_plan(int64_t M, int64_t N, int64_t K, ClusterPlan *out) {
    if (M < 1 || N < 1 || K < 1 || M > 148 * kCMaxT || N > 148ll * kCUnitN) return false;
    const int sms = sm_count();
    const int tiles_n = static_cast<int>((N + kCUnitN - 1) / kCUnitN), num_kb = static_cast<int>((K + kCBK - 1) / kCBK);
    const int rows = static_cast<int>(M);
    const float memory = (static_cast<float>(K) * N + static_cast<float>(M) * K + 2.0f * M * N) / 6500.0f;
    float best = 0.0f;
    bool two = false;
    for (int T = 32; T <= kCMaxT; T += 32) {
        const int tiles = (rows + T - 1) / T;
        if (T > 32 && (rows + T - 33) / (T - 32) == tiles) continue;  // a lower tile gives as many
        const float bytes = kCWBytes + T * (kCBK / 2);
        const float block = std::max(bytes / 105.0f, 1.4f * T);
        for (int s = 0, slices = 1; slices <= 4 && slices <= num_kb; ++s, slices *= 2) {
            const int resident = s == 0 ? sms / 2 : s == 1 ? sms * 33 / 148 : sms * 15 / 148;
            const int64_t clusters = static_cast<int64_t>(tiles_n) * tiles;
            if (clusters > 2 * resident) continue;
            const bool twice = clusters > resident;
            const int blocks = (num_kb + slices - 1) / slices;
            const float loop = blocks * block * (twice ? 2 : 1), l2 = clusters * 2.0f * slices * blocks * bytes / 14000.0f;
            const float exchange = slices == 1 ? 0.0f : (slices == 2 ? 1200.0f : 2400.0f) + 12.0f * T;
            const float cost = std::max(std::max(loop, l2), memory) + exchange + 4.0f * T / slices * (twice ? 2 : 1);
            if (out->T != 0 && cost >= best) continue;
            // the ring receives the other slices' sums (256 tokens over four slices with two CTAs an SM fill all of it)
            const int stage_bytes = kCWBytes + T / 2 * kCBK;
            if ((slices - 1) * (T / slices) * (kCUnitN / 2) * 4 > cluster_stages(stage_bytes, twice) * stage_bytes) continue;
            best = cost;
            two = twice;
            out->T = T;
            out->slices = slices;
            out->clusters = clusters;
        }
    }
    if (out->T == 0) return false;
    out->stage_bytes = kCWBytes + out->T / 2 * kCBK;
    out->stages = cluster_stages(out->stage_bytes, two);
    out->smem = static_cast<size_t>(out->stages) * out->stage_bytes + sizeof(ClusterSmemTail);
    while (out->tmem_cols < static_cast<uint32_t>(out->T)) out->tmem_cols *= 2;
    return true;
}

template <typename OutT>
int launch_cluster_t(const int8_t *x1, int64_t ld_x1, const int8_t *x2, int64_t x2_sk, int64_t x2_sn, const EpilogueParams &ep,
                     int64_t K, const ClusterPlan &pl, cudaStream_t stream) {
    ClusterParams p;
    p.ep = ep;
    p.num_kb = static_cast<int>((K + kCBK - 1) / kCBK);
    p.T = pl.T;
    p.tiles_m = static_cast<int>((ep.M + pl.T - 1) / pl.T);
    p.stages = pl.stages;
    p.stage_bytes = pl.stage_bytes;
    p.tmem_cols = pl.tmem_cols;
    p.status = device_status_word();
    const bool mn_major = (x2_sn == 1);
    CUtensorMap tw, tx;
    int rc;
    if (mn_major)
        rc = make_tmap_2d(&tw, x2, 1, static_cast<uint64_t>(ep.N), static_cast<uint64_t>(K), static_cast<uint64_t>(x2_sk),
                          kCUnitN / 2, kCBK, true);
    else
        rc = make_tmap_2d(&tw, x2, 1, static_cast<uint64_t>(K), static_cast<uint64_t>(ep.N), static_cast<uint64_t>(x2_sn), kCBK,
                          kCUnitN / 2, true);
    if (rc != QMM_OK) return rc;
    rc = make_tmap_2d(&tx, x1, 1, static_cast<uint64_t>(K), static_cast<uint64_t>(ep.M), static_cast<uint64_t>(ld_x1), kCBK,
                      static_cast<uint32_t>(pl.T / 2), true);
    if (rc != QMM_OK) return rc;
    using Kernel = void (*)(CUtensorMap, CUtensorMap, ClusterParams);
    const Kernel kern = pl.slices == 1   ? (mn_major ? w8a8_cluster_kernel<OutT, true, 1> : w8a8_cluster_kernel<OutT, false, 1>)
                        : pl.slices == 2 ? (mn_major ? w8a8_cluster_kernel<OutT, true, 2> : w8a8_cluster_kernel<OutT, false, 2>)
                                         : (mn_major ? w8a8_cluster_kernel<OutT, true, 4> : w8a8_cluster_kernel<OutT, false, 4>);
    QMM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kCMaxSmem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(pl.clusters * 2 * pl.slices));
    cfg.blockDim = dim3(kCThreads);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(2 * pl.slices);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    QMM_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tw, tx, p));
    return QMM_OK;
}

}  // namespace

bool prefer_cluster(int64_t M, int64_t N, int64_t K) {
    ClusterPlan pl;
    if (!cluster_make_plan(M, N, K, &pl)) return false;
    const int64_t num_kb = (K + kCBK - 1) / kCBK;
    // so few columns and so long a K that four slices leave a CTA a long chain: stream-K (M x K x N = 1 x 28672 x 512 9.0 us,
    // here 10.9; 8 x 28672 x 1024 10.8 / 11.6; 16 x 28672 x 1024 12.2 / 11.6; 8 x 16384 x 1024 10.0 / 8.0)
    if (M <= 8 && N <= 4 * kCUnitN && num_kb > 176) return false;
    // tiles of 256 x 256 either way: the persistent kernel computes one while it stores the one before (us, here / there:
    // 512 x 4096 x 14336 29.0 / 26.9, 2048 x 4096 x 4096 28.6 / 26.7, 1024 x 1024 x 4096 9.9 / 9.4, 2048 x 14336 x 4096 77.9 / 77.2;
    // 640 x 4096 x 8192, three lower tiles here, 19.8 / 25.9).  Lower tiles stay here, also those with two an SM on some SMs and one on
    // others.  Time here over there, least, median and most of 75 to 148 clusters of one slice, K of 1024 to 28672, 16-bit and int32
    // outputs, both weight layouts: 160 tokens a tile 0.64 0.83 1.00, 192 0.72 0.88 1.03, 224 0.80 0.94 1.10 (about even with 16-bit outputs
    // for K up to 3072, and for a long K where a row of the operands is no multiple of 128 bytes).
    if (M > 128 && pl.T == kCMaxT && pl.slices == 1) return false;
    return true;
}

int launch_cluster(const int8_t *x1, int64_t ld_x1, const int8_t *x2, int64_t x2_sk, int64_t x2_sn, const EpilogueParams &ep,
                   int out_dtype, int64_t K, cudaStream_t stream) {
    ClusterPlan pl;
    if (!cluster_make_plan(ep.M, ep.N, K, &pl))
        return fail(QMM_ERR_UNSUPPORTED, "qmm_quant_matmul: the cluster kernel needs tiles of 256 columns x up to 256 tokens that "
                                         "are all resident at once");
    switch (out_dtype) {
        case QMM_DTYPE_BF16:
            return launch_cluster_t<__nv_bfloat16>(x1, ld_x1, x2, x2_sk, x2_sn, ep, K, pl, stream);
        case QMM_DTYPE_F16:
            return launch_cluster_t<__half>(x1, ld_x1, x2, x2_sk, x2_sn, ep, K, pl, stream);
        case kOutI8:
            return launch_cluster_t<int8_t>(x1, ld_x1, x2, x2_sk, x2_sn, ep, K, pl, stream);
        default:
            return launch_cluster_t<int32_t>(x1, ld_x1, x2, x2_sk, x2_sn, ep, K, pl, stream);
    }
}

}  // namespace qmm
