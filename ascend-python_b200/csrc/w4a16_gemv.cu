// W4A16 matmul for one or two tokens over prepacked weights: integer dot products on the CUDA cores.
//
// For so few tokens the tensor cores have nothing to add: a thread owns one output column, reads its 64 bytes of a block (of the
// stream of w4a16_prepacked.cu: 128 columns x 128 k, 8704 bytes), splits each packed word into two words of four unsigned
// bytes - `w ^ 0x88888888` turns the two's complement nibbles into w + 8, `& 0x0f0f0f0f` and `>> 4 & 0x0f0f0f0f` are bytes
// (k, k+4, k+1, k+5) and (k+2, k+6, k+3, k+7) of a group of eight k - and multiplies them with dp4a by the activations as two
// int8 digits of a block floating-point form, in that byte order: per token and block of 128 k, with e the exponent of the
// block's absmax,
//     X = rint(x * 2^(14 - e))  (|X| <= 2^14),   X = 128 * d1 + d2,  d1 in [-128, 127], d2 in [0, 127].
// An activation within 2^-6 of its block's absmax is represented exactly (16-bit floats carry 8 or 11 significant bits); smaller
// ones are rounded to 2^-14 of the absmax, far below the 2^-9 / 2^-12 of the output's own rounding.  Per block the exact
// integers D1 = sum u*d1 and D2 = sum u*d2 (u = w + 8) give
//     y[m, n] += scale * esc[m] * (128 D1 + D2) + (offset*scale - 8 scale) * xs[m],
// esc = 2^(e - 14), xs = esc * sum X; the weight itself is never rounded.
//
// A CTA works on one tile of 128 columns and a slice of K; the slices of a tile are the CTAs of a cluster.  One thread streams
// the slice's blocks, which are contiguous, into a ring in shared memory by bulk copies; meanwhile the others make the digits of
// the slice; then three groups of 128 threads take the blocks in turn.  Their sums meet in shared memory, the slices' in the
// first CTA's, in their order: results do not depend on timing, and there is no scratch, no counter and no second kernel.
#include <algorithm>

#include "qmm_common.cuh"
#include "w4a16_gemv.cuh"

namespace qmm {

namespace {

constexpr int kVTileN = 128;
constexpr int kVBlockK = 128;
constexpr int kVSubs = 4;                                 // sub-steps of 32 k of a block
constexpr int kVWBytes = kVTileN * kVBlockK / 2;          // 8192
constexpr int kVBlockBytes = kVWBytes + 2 * kVTileN * 2;  // 8704
constexpr int kVGroups = 3;
constexpr int kVWarps = kVGroups * kVTileN / 32;          // that take blocks
constexpr int kVThreads = (kVWarps + 1) * 32;
constexpr int kVMaxRing = 15;
constexpr int kVMaxSmem = 220 * 1024;
static_assert(kVMaxRing % kVGroups == 0, "see v_make_plan");

struct VSmemTail {
    uint64_t full[kVMaxRing];
    uint64_t empty[kVMaxRing];
    uint32_t abort_flag;
};

struct VParams {
    const uint8_t *packed;
    const void *x;
    int64_t ld_x;
    const void *bias;
    void *out;
    int64_t ld_out;
    int M, N, nblocks;  // blocks of 128 k, rounded up to an even number
    int64_t K;
    int slices, ring, max_blocks;  // most blocks of a slice
    uint32_t *status;
};

__device__ __forceinline__ void v_consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kVWarps * 32) : "memory"); }
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// A lane's four consecutive activations of token m's block of 128 k; zeros beyond (K is a multiple of 128: a block is inside or a
// padding block).
template <typename T>
__device__ __forceinline__ uint2 v_load_x(const VParams &p, int m, int blk) {
    const int64_t k0 = static_cast<int64_t>(blk) * kVBlockK + (threadIdx.x & 31) * 4;
    return k0 < p.K ? __ldg(reinterpret_cast<const uint2 *>(static_cast<const T *>(p.x) + m * p.ld_x + k0)) : make_uint2(0, 0);
}

// Digits of those of a warp.  rec: 256 bytes, d1 then d2.
template <typename T>
__device__ __forceinline__ void v_make_digits(uint2 raw, uint8_t *rec, float *esc, float *xs) {
    const int lane = threadIdx.x & 31;
    const T *h = reinterpret_cast<const T *>(&raw);
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = to_float(h[j]);
    float a = 0.0f;
    int bad = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float av = fabsf(v[j]);
        if (av <= 3.0e38f) a = fmaxf(a, av); else bad = 1;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
    bad = __any_sync(0xffffffffu, bad);
    int e = 0, sum = 0;
    float e_scale = 0.0f;
    if (a > 0.0f) {
        (void)frexpf(a, &e);  // a = f * 2^e, f in [0.5, 1): |x| < 2^e; X = rint(x * 2^(14 - e))
        e_scale = ldexpf(1.0f, e - 14);
    }
    // the four k of a lane lie in one group of eight, whose two words are bytes [8 i, 8 i + 8) of the sub-step's 32
    const int s = lane >> 3, i = (lane >> 1) & 3;
    uint32_t d1w[2] = {0, 0}, d2w[2] = {0, 0};  // this lane's bytes of the group's two words
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
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) {
        // a block that holds a NaN or an infinity poisons the token's outputs
        *esc = bad ? __int_as_float(0x7fc00000) : e_scale;
        *xs = e_scale * static_cast<float>(sum);  // |sum| < 2^21: exact
    }
}

template <typename T, int M>
__global__ void __launch_bounds__(kVThreads, 2)
w4a16_gemv_tile_kernel(VParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    // [ring of blocks][digits [block][M][256]][esc [block][M]][xs [block][M]][groups' sums [3][M][128]][slices' sums][tail]
    uint8_t *digits = smem + p.ring * kVBlockBytes;
    float *esc = reinterpret_cast<float *>(digits + p.max_blocks * M * 256);
    float *xs = esc + p.max_blocks * M;
    float *other = xs + p.max_blocks * M;
    float *recv = other + kVGroups * M * kVTileN;
    VSmemTail *tail = reinterpret_cast<VSmemTail *>(recv + (p.slices - 1) * M * kVTileN);
    volatile uint32_t *abort_flag = &tail->abort_flag;
    pdl_launch_dependents();
    // distributed shared memory is written only when every CTA of the cluster has started: see the wait below
    if (p.slices > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

    const int warp = warp_id_uniform(), lane = threadIdx.x & 31;
    const int tile = static_cast<int>(blockIdx.x) / p.slices, slice = static_cast<int>(blockIdx.x) % p.slices;
    const int b_begin = static_cast<int>(static_cast<int64_t>(p.nblocks) * slice / p.slices);
    const int nb = static_cast<int>(static_cast<int64_t>(p.nblocks) * (slice + 1) / p.slices) - b_begin;
    const uint32_t ring = static_cast<uint32_t>(p.ring);
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < ring; ++s) {
            mbar_init(smem_u32(&tail->full[s]), 1);
            mbar_init(smem_u32(&tail->empty[s]), kVTileN / 32);
        }
        tail->abort_flag = 0;
        mbar_fence_init();
    }
    pdl_wait();
    __syncthreads();

    const int64_t n = static_cast<int64_t>(tile) * kVTileN + threadIdx.x;  // the first four warps finish a column a thread
    const bool finisher = threadIdx.x < kVTileN;

    if (warp == kVWarps) {
        // ---------------- the stream of blocks ----------------
        const uint8_t *src = p.packed + (static_cast<int64_t>(tile) * p.nblocks + b_begin) * kVBlockBytes;
        uint32_t st = 0, ph = 0;
        for (int b = 0; b < nb; ++b, src += kVBlockBytes) {
            if (!mbar_wait(smem_u32(&tail->empty[st]), ph ^ 1, abort_flag, 0x81)) break;
            if (lane == 0) {
                const uint32_t bar = smem_u32(&tail->full[st]);
                mbar_expect_tx(bar, kVBlockBytes);
                bulk_load_1d(smem_u32(smem) + st * kVBlockBytes, src, kVBlockBytes, bar);
            }
            __syncwarp();
            if (++st == ring) {
                st = 0;
                ph ^= 1;
            }
        }
    } else {
        // six loads under way at a time (1 x 7680 x 19200, whose tiles are one slice each, has five a warp)
        for (int i0 = warp; i0 < nb * M; i0 += 6 * kVWarps) {
            uint2 raw[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const int i = i0 + j * kVWarps;
                raw[j] = i < nb * M ? v_load_x<T>(p, i % M, b_begin + i / M) : make_uint2(0, 0);
            }
#pragma unroll 1
            for (int j = 0; j < 6; ++j) {
                const int i = i0 + j * kVWarps;
                if (i >= nb * M) break;
                const uint2 v = raw[0];
#pragma unroll
                for (int q = 0; q < 5; ++q) raw[q] = raw[q + 1];
                v_make_digits<T>(v, digits + i * 256, esc + i, xs + i);
            }
        }
        v_consumer_sync();
        const int r = threadIdx.x & (kVTileN - 1), group = warp / (kVTileN / 32);
        float y[M];
#pragma unroll
        for (int m = 0; m < M; ++m) y[m] = 0.0f;
        uint32_t st = static_cast<uint32_t>(group), ph = 0;  // the ring is a multiple of the groups: a slot is always one group's
        for (int b = group; b < nb; b += kVGroups) {
            if (!mbar_wait(smem_u32(&tail->full[st]), ph, abort_flag, 0x82)) break;
            const uint8_t *blk = smem + st * kVBlockBytes;
            uint4 wv[kVSubs];
#pragma unroll
            for (int s = 0; s < kVSubs; ++s) wv[s] = *reinterpret_cast<const uint4 *>(blk + (s * kVTileN + r) * 16);
            const float sc = to_float(*reinterpret_cast<const T *>(blk + kVWBytes + r * 2));
            const float tc = to_float(*reinterpret_cast<const T *>(blk + kVWBytes + kVTileN * 2 + r * 2)) - 8.0f * sc;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tail->empty[st]));
            int d1[M], d2[M];
#pragma unroll
            for (int m = 0; m < M; ++m) d1[m] = d2[m] = 0;
            const uint4 *xd = reinterpret_cast<const uint4 *>(digits) + b * M * 16;
#pragma unroll
            for (int s = 0; s < kVSubs; ++s) {
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
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const float v = fmaf(static_cast<float>(d1[m]), 128.0f, static_cast<float>(d2[m]));
                y[m] = fmaf(sc * esc[b * M + m], v, y[m]);
                y[m] = fmaf(tc, xs[b * M + m], y[m]);
            }
            st += kVGroups;
            if (st >= ring) {
                st -= ring;
                ph ^= 1;
            }
        }
#pragma unroll
        for (int m = 0; m < M; ++m) other[(group * M + m) * kVTileN + r] = y[m];
        v_consumer_sync();
    }
    __syncwarp();
    float sum[M];
    if (finisher) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            sum[m] = 0.0f;
#pragma unroll
            for (int g = 0; g < kVGroups; ++g) sum[m] += other[(g * M + m) * kVTileN + threadIdx.x];
        }
    }
    if (p.slices > 1) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        // a slice that was cut short sends what it has: the status word tells
        if (finisher && slice != 0) {
#pragma unroll
            for (int m = 0; m < M; ++m)
                st_cluster_f32(map_to_cta(smem_u32(recv + ((slice - 1) * M + m) * kVTileN + threadIdx.x), 0), sum[m]);
        }
        cluster_sync_all();
        if (finisher && slice == 0) {
            for (int s = 0; s < p.slices - 1; ++s)
#pragma unroll
                for (int m = 0; m < M; ++m) sum[m] += recv[(s * M + m) * kVTileN + threadIdx.x];
        }
    }
    if (finisher && slice == 0 && n < p.N) {
        const float bias = p.bias != nullptr ? to_float(static_cast<const T *>(p.bias)[n]) : 0.0f;
#pragma unroll
        for (int m = 0; m < M; ++m) static_cast<T *>(p.out)[m * p.ld_out + n] = from_float<T>(sum[m] + bias);
    }
    if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) atomicMax(p.status, *abort_flag);
}

struct VPlan {
    int slices = 0, ring = 0, max_blocks = 0;
    size_t smem = 0;
};

size_t v_fixed_bytes(int m, int max_blocks, int slices) {
    return static_cast<size_t>(max_blocks) * m * (256 + 8) + static_cast<size_t>(kVGroups + slices - 1) * m * kVTileN * sizeof(float) +
           sizeof(VSmemTail);
}

constexpr int kVMaxSlices = 8;

cudaLaunchConfig_t v_launch_config(int64_t ctas, int slices, size_t smem, cudaStream_t stream, cudaLaunchAttribute (&attr)[2]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(kVThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(slices);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

// Clusters of each size that are resident at once, with one CTA an SM and with two (a cluster lies within a GPC, so this is less
// than the SMs divided by the size).
struct VResident {
    int one[kVMaxSlices + 1], two[kVMaxSlices + 1];
};
const VResident &v_resident() {
    static const VResident r = [] {
        VResident v;
        const auto kern = w4a16_gemv_tile_kernel<__half, 1>;
        const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kVMaxSmem) == cudaSuccess;
        for (int s = 0; s <= kVMaxSlices; ++s) {
            v.one[s] = v.two[s] = 0;
            if (s < 2 || !ok) continue;  // one CTA a tile: no cluster
            cudaLaunchAttribute attr[2];
            cudaLaunchConfig_t cfg = v_launch_config(s, s, kVMaxSmem, nullptr, attr);
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&v.one[s], kern, &cfg) != cudaSuccess) v.one[s] = 0;
            cfg.dynamicSmemBytes = kVMaxSmem / 2;
            if (cudaOccupancyMaxActiveClusters(&v.two[s], kern, &cfg) != cudaSuccess) v.two[s] = 0;
        }
        (void)cudaGetLastError();
        return v;
    }();
    return r;
}

// Slices of K by a model of the time, in clocks: a block takes an SM 256 for each token (dp4a), and all SMs together get a block
// every 2.6 from memory; a CTA alone on an SM takes 1.3 times that.  Clusters that are not resident at once are not considered
// (37 tiles: four slices, of which 33 clusters fit with one CTA an SM, 9.7 us for one token of 10624 x 4680, three slices 7.1).
// The ring: as many blocks as fit beside the digits.
bool v_make_plan(int m, int64_t N, int64_t K, VPlan *pl) {
    const int64_t tiles = (N + kVTileN - 1) / kVTileN, blocks = (K + 2 * kVBlockK - 1) / (2 * kVBlockK) * 2;
    const int sms = sm_count();
    if (blocks > (1 << 20)) return false;
    float best = 0.0f;
    pl->slices = 0;
    for (int slices = 1; slices <= kVMaxSlices; ++slices) {
        if (slices > 1 && (blocks < 4 * slices || tiles > v_resident().two[slices])) continue;
        const int64_t most = (blocks + slices - 1) / slices;
        const int64_t one = slices == 1 ? sms : v_resident().one[slices], an_sm = slices == 1 ? (tiles + sms - 1) / sms : tiles > one ? 2 : 1;
        const size_t fixed = v_fixed_bytes(m, static_cast<int>(most), slices);
        size_t budget = an_sm > 1 ? kVMaxSmem / 2 : kVMaxSmem;
        if (slices == 1 && fixed + 2 * kVGroups * kVBlockBytes > budget) budget = kVMaxSmem;
        if (fixed + 2 * kVGroups * kVBlockBytes > budget) continue;
        const float busy = std::min(1.0f, static_cast<float>(tiles * slices) / static_cast<float>(sms));
        const float cost = static_cast<float>(most * an_sm) * std::max(256.0f * m, 390.0f * busy) * (an_sm > 1 ? 1.0f : 1.3f) +
                           (slices > 1 ? 600.0f + 60.0f * slices : 0.0f);
        if (pl->slices != 0 && cost >= best) continue;
        best = cost;
        pl->slices = slices;
        pl->max_blocks = static_cast<int>(most);
        // A multiple of the groups.  Otherwise blocks of different groups follow one another in a slot, and a group that is ahead
        // could test its phase of the slot's barrier before the phase in front has completed, which parity cannot tell apart.
        const int fit = static_cast<int>((budget - fixed) / kVBlockBytes) / kVGroups * kVGroups;
        const int need = static_cast<int>((most + kVGroups - 1) / kVGroups * kVGroups);
        pl->ring = std::min({need, kVMaxRing, fit});
        pl->smem = fixed + static_cast<size_t>(pl->ring) * kVBlockBytes;
    }
    return pl->slices != 0;
}

template <typename T>
int launch_gemv_tile_t(VParams &p, const VPlan &pl, int64_t tiles, cudaStream_t stream) {
    using Kernel = void (*)(VParams);
    const Kernel kern = p.M == 1 ? w4a16_gemv_tile_kernel<T, 1> : w4a16_gemv_tile_kernel<T, 2>;  // kGemvMaxM
    QMM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kVMaxSmem));
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = v_launch_config(tiles * pl.slices, pl.slices, pl.smem, stream, attr);
    if (pl.slices == 1) {  // no cluster
        cfg.attrs = attr + 1;
        cfg.numAttrs = 1;
    }
    QMM_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, p));
    return QMM_OK;
}

}  // namespace

// Compute bounds it from some size on: the digits' dp4a issue at 32 lanes a clock, 13 us a token for 8192 x 28672, and where a
// weight has more tiles than there are SMs those with two take twice that.  The kernel of w4a16_prepacked.cu deals out the
// blocks evenly, but pays for a kernel in front, scratch, counters and a last arrival.  us, there / here (K x N): one token
// 1024 x 1024 5.1 / 3.0, 4096 x 4096 9.2 / 5.1, 8192 x 8192 13.4 / 8.7, 4096 x 28672 16.7 / 13.4, 28672 x 8192 25.4 / 23.2,
// 8192 x 28672 25.4 / 24.8
// (25.9 / 26.5 with other launches between), 28672 x 28672 72 / 84; two tokens 4096 x 4096 10.6 / 7.1, 8192 x 8192 16.1 / 12.1, 4096 x 28672
// 20.0 / 20.9, 8192 x 28672 31.9 / 38.9.
bool prefer_gemv_tile(int64_t M, int64_t N, int64_t K) {
    VPlan pl;
    const bool one_wave = N <= static_cast<int64_t>(sm_count()) * kVTileN;
    return M >= 1 && M <= kGemvMaxM && K <= (M == 2 ? 75000000 : one_wave ? 300000000 : 150000000) / N &&
           v_make_plan(static_cast<int>(M), N, K, &pl);
}

int launch_gemv_tile(const void *packed, const void *x, int x_dtype, int64_t ld_x, const void *bias, void *out, int64_t ld_out,
                     int64_t M, int64_t N, int64_t K, cudaStream_t stream) {
    VPlan pl;
    if (M < 1 || M > kGemvMaxM || !v_make_plan(static_cast<int>(M), N, K, &pl))
        return fail(QMM_ERR_UNSUPPORTED, "w4a16: the activations' digits do not fit in shared memory");
    VParams p;
    p.packed = static_cast<const uint8_t *>(packed);
    p.x = x;
    p.ld_x = ld_x;
    p.bias = bias;
    p.out = out;
    p.ld_out = ld_out;
    p.M = static_cast<int>(M);
    p.N = static_cast<int>(N);
    p.K = K;
    p.nblocks = static_cast<int>((K + 2 * kVBlockK - 1) / (2 * kVBlockK)) * 2;
    p.slices = pl.slices;
    p.ring = pl.ring;
    p.max_blocks = pl.max_blocks;
    p.status = device_status_word();
    const int64_t tiles = (N + kVTileN - 1) / kVTileN;
    return x_dtype == QMM_DTYPE_BF16 ? launch_gemv_tile_t<__nv_bfloat16>(p, pl, tiles, stream)
                                     : launch_gemv_tile_t<__half>(p, pl, tiles, stream);
}

}  // namespace qmm
