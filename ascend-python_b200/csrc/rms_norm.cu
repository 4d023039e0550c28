// RMS normalisation (npu_rms_norm) and its fusion with the per-token dynamic quantization that
// follows it in a decoder block (npu_rms_norm_dynamic_quant).
//
// Reference: op_plugin/ops/base_ops/opapi/RmsNormKernelOpApi.cpp:24-35 (host function: outputs y with
// the input's dtype and rstd in fp32) and the numpy golden of
// test/test_custom_ops/test_npu_rms_norm.py:10-18:
//     variance = mean(x^2, axis=-1);  rstd = 1 / sqrt(variance + epsilon);  y = (x * rstd) * gamma
// All arithmetic is fp32 with one rounding per operation in that order; y is rounded once to the
// input dtype.  The sum of squares is taken per thread over its elements in index order, then over
// the lanes of a warp by an xor-shuffle tree, then over the warps of a row in warp order, so it does
// not depend on timing.
//
// One pass over HBM: a row stays in registers as 128-bit vectors between the reduction and the
// scaling.  The fused kernel goes on in the same registers: absmax of the ROUNDED y, scale =
// amax / 127, q = rint(y / scale), exactly the arithmetic of qmm_dynamic_quant applied to the y that
// qmm_rms_norm would have stored, so fused and unfused results are identical bit for bit while y
// never travels to HBM and back (2 * cols bytes written + 2 * cols bytes read per row saved).
#include <type_traits>

#include "dynamic_quant.cuh"

namespace qmm {

namespace {

using dq::max_nan;

template <typename T>
struct VecOf {
    static constexpr int kElems = 16 / sizeof(T);
};

template <typename T>
__device__ __forceinline__ void unpack_vec(const uint4 &v, float (&f)[VecOf<T>::kElems]);
template <>
__device__ __forceinline__ void unpack_vec<float>(const uint4 &v, float (&f)[4]) {
    f[0] = __uint_as_float(v.x);
    f[1] = __uint_as_float(v.y);
    f[2] = __uint_as_float(v.z);
    f[3] = __uint_as_float(v.w);
}
template <>
__device__ __forceinline__ void unpack_vec<__nv_bfloat16>(const uint4 &v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
template <>
__device__ __forceinline__ void unpack_vec<__half>(const uint4 &v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 p = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        f[2 * i] = p.x;
        f[2 * i + 1] = p.y;
    }
}

template <typename T>
__device__ __forceinline__ uint4 pack_vec(const float (&f)[VecOf<T>::kElems]);
template <>
__device__ __forceinline__ uint4 pack_vec<float>(const float (&f)[4]) {
    return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
}
template <>
__device__ __forceinline__ uint4 pack_vec<__nv_bfloat16>(const float (&f)[8]) {
    return make_uint4(pack2<__nv_bfloat16>(f[0], f[1]), pack2<__nv_bfloat16>(f[2], f[3]),
                      pack2<__nv_bfloat16>(f[4], f[5]), pack2<__nv_bfloat16>(f[6], f[7]));
}
template <>
__device__ __forceinline__ uint4 pack_vec<__half>(const float (&f)[8]) {
    return make_uint4(pack2<__half>(f[0], f[1]), pack2<__half>(f[2], f[3]), pack2<__half>(f[4], f[5]),
                      pack2<__half>(f[6], f[7]));
}

__device__ __forceinline__ float rstd_of(float sumsq, int cols, float eps) {
    const float variance = __fdiv_rn(sumsq, static_cast<float>(cols));
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(variance, eps)));
}

// Columns [c, c + 8) of gamma, whose vectors are aligned where c is a multiple of eight, for a row that is shifted against
// them by c mod 8 elements (the same for all threads of a row): two vectors and a funnel shift.
template <typename T>
__device__ __forceinline__ uint4 load_gamma_shifted(const T *gamma, int c, int cols) {
    const int s = c & 7;
    const uint4 a = dq::load8_edge(gamma, c - s, cols);
    if (s == 0) return a;
    const uint4 b = dq::load8_edge(gamma, c - s + 8, cols);
    const bool far = (s & 4) != 0, odd = (s & 2) != 0;
    uint32_t w[6] = {far ? a.z : a.x, far ? a.w : a.y, far ? b.x : a.z, far ? b.y : a.w, far ? b.z : b.x, far ? b.w : b.y};
#pragma unroll
    for (int j = 0; j < 5; ++j) w[j] = odd ? w[j + 1] : w[j];
    const uint32_t bits = (s & 1) * 16;
    return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits), __funnelshift_r(w[2], w[3], bits),
                      __funnelshift_r(w[3], w[4], bits));
}

// `tpr` threads per row, each holding VPT 16-byte vectors.  QUANT: write int8 + scale instead of y.  SHIFTED: 16-bit rows
// that begin off the vector grid (see dynamic_quant.cuh).
template <typename T, int VPT, bool QUANT, bool SHIFTED = false>
__global__ void __launch_bounds__(512)
rms_norm_vec_kernel(const T *__restrict__ x, int64_t rows, int cols, int64_t ld_x, const T *__restrict__ gamma,
                    float eps, T *__restrict__ y, int64_t ld_y, int8_t *__restrict__ q, int64_t ld_q,
                    float *__restrict__ scale, float *__restrict__ rstd_out, int tpr) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int E = VecOf<T>::kElems;
    __shared__ float s_part[2][16];
    const int tpr_shift = __ffs(tpr) - 1;  // tpr is a power of two
    const int rows_per_cta = blockDim.x >> tpr_shift;
    const int row_in_cta = threadIdx.x >> tpr_shift;
    const int t = threadIdx.x & (tpr - 1);
    const int64_t row = static_cast<int64_t>(blockIdx.x) * rows_per_cta + row_in_cta;
    const bool row_ok = row < rows;
    const int shift = SHIFTED ? dq::row_shift(x + row * ld_x) : 0;
    const int nvec = (SHIFTED ? cols + shift + E - 1 : cols) / E;
    const int warp = threadIdx.x >> 5;
    const int warps_per_row = tpr >> 5;
    const int w0 = row_in_cta * warps_per_row;

    uint4 v[VPT];
    float sumsq = 0.0f;
    if (row_ok) {
        const T *src = x + row * ld_x;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int idx = t + i * tpr;
            v[i] = make_uint4(0, 0, 0, 0);
            if (idx < nvec) {
                if constexpr (SHIFTED)
                    v[i] = dq::load8_edge(src, idx * E - shift, cols);
                else
                    v[i] = __ldg(reinterpret_cast<const uint4 *>(src) + idx);
            }
        }
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            float f[E];
            unpack_vec<T>(v[i], f);
#pragma unroll
            for (int j = 0; j < E; ++j) sumsq = fmaf(f[j], f[j], sumsq);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sumsq += __shfl_xor_sync(0xffffffffu, sumsq, o);
    if (tpr > 32) {
        if ((threadIdx.x & 31) == 0) s_part[0][warp] = sumsq;
        __syncthreads();
        float s = 0.0f;
        for (int w = 0; w < warps_per_row; ++w) s += s_part[0][w0 + w];
        sumsq = s;
    }
    const float rstd = rstd_of(sumsq, cols, eps);
    if (row_ok && t == 0) rstd_out[row] = rstd;

    // y = (x * rstd) * gamma, rounded once to T; kept in the same registers
    float amax = 0.0f;
    if (row_ok) {
        const uint4 *gsrc = reinterpret_cast<const uint4 *>(gamma);
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int idx = t + i * tpr;
            if (idx < nvec) {
                float f[E], g[E];
                unpack_vec<T>(v[i], f);
                if constexpr (SHIFTED)
                    unpack_vec<T>(load_gamma_shifted(gamma, idx * E - shift, cols), g);
                else
                    unpack_vec<T>(__ldg(gsrc + idx), g);
#pragma unroll
                for (int j = 0; j < E; ++j) f[j] = __fmul_rn(__fmul_rn(f[j], rstd), g[j]);
                v[i] = pack_vec<T>(f);
                if constexpr (QUANT) {
                    amax = max_nan(amax, dq::absmax8<T>(v[i]));  // of the rounded values
                } else if constexpr (SHIFTED) {
                    dq::store8_edge(y + row * ld_y, idx * E - shift, cols, v[i]);
                } else {
                    reinterpret_cast<uint4 *>(y + row * ld_y)[idx] = v[i];
                }
            }
        }
    }
    if constexpr (QUANT) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (tpr > 32) {
            if ((threadIdx.x & 31) == 0) s_part[1][warp] = amax;
            __syncthreads();
            float m = 0.0f;
            for (int w = 0; w < warps_per_row; ++w) m = max_nan(m, s_part[1][w0 + w]);
            amax = m;
        }
        if (!row_ok) return;
        const dq::RowQuant rq = dq::make_row_quant(amax);
        if (t == 0) scale[row] = rq.scale;
        const bool fast = !rq.exact_only && rq.scale != 0.0f;
        int8_t *dst = q + row * ld_q;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int idx = t + i * tpr;
            if (idx < nvec) {
                float f[8];
                dq::unpack8<T>(v[i], f);
                const uint2 b = dq::quantize8(f, rq, fast);
                if constexpr (SHIFTED)
                    dq::store8_edge(dst, idx * E - shift, cols, b);
                else
                    reinterpret_cast<uint2 *>(dst)[idx] = b;
            }
        }
    }
}

// The fused kernel for rows of up to 256 threads: a CTA walks rows.  FULL: the row fills all vectors (cols == tpr * VPT *
// 8), no guards.  With one row per CTA and scalar arithmetic (the kernel above) it was bound by instruction issue: 20
// instructions an element, 30.8 us at 8192 x 4096 where the memory needs 15.  So the fp32 arithmetic is two
// elements an instruction where its order allows, guards and the choice of quantizer are outside the loops over
// elements, there is a variant for every number of vectors, and the next row's loads are under way while a row is
// worked on (its registers are free as soon as the row is unpacked).  8192 x 4096: 25.7 us, 16 instructions an element at
// 63 % of the issue slots: 128 registers leave 16 warps an SM, too few to fill the rest; 8192 x 8192: 50.6 -> 45.8;
// 4096 x 16384: 52.1 -> 47.8; 4096 x 5128: 20.4 -> 18.9.  Rows of 512 threads leave one CTA an SM and nothing to overlap
// its barriers with (1000 x 30000: 30.1 us against 28.0): they stay with the kernel above, and so does the plain
// operator, which is close to the memory's rate.  The sum of squares is taken in that kernel's order.
// SHIFTED: rows that begin off the vector grid (see dynamic_quant.cuh); gamma is then read again for every row.
template <typename T, int VPT, bool FULL, bool SHIFTED = false>
__global__ void __launch_bounds__(256, 2)
rms_norm_quant_walk_kernel(const T *__restrict__ x, int64_t rows, int cols, int64_t ld_x, const T *__restrict__ gamma,
                    float eps, int8_t *__restrict__ q, int64_t ld_q,
                    float *__restrict__ scale, float *__restrict__ rstd_out, int tpr) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int E = VecOf<T>::kElems, H = E / 2;
    static_assert(E == 8, "16-bit types");
    constexpr bool kKeepGamma = VPT * E <= 32 && !SHIFTED;
    __shared__ float s_part[2][2][8];  // [row parity][sum, absmax][warp]
    const int tpr_shift = __ffs(tpr) - 1;
    const int rows_per_cta = blockDim.x >> tpr_shift;
    const int row_in_cta = threadIdx.x >> tpr_shift;
    const int t = threadIdx.x & (tpr - 1);
    int64_t row = static_cast<int64_t>(blockIdx.x) * rows_per_cta + row_in_cta;
    int shift = 0, nvec = cols / E;  // of the row that is worked on
    auto set_shift = [&](int64_t r) {
        if constexpr (SHIFTED) {
            shift = dq::row_shift(x + r * ld_x);
            nvec = (cols + shift + E - 1) / E;
        }
    };
    set_shift(row);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warps_per_row = tpr >> 5;
    const int w0 = row_in_cta * warps_per_row;
    auto has = [&](int i) { return FULL || t + i * tpr < nvec; };

    float2 g[kKeepGamma ? VPT : 1][H];
    auto load_gamma = [&](int i, float2 (&out)[H]) {
        float f[E];
        if constexpr (SHIFTED)
            unpack_vec<T>(has(i) ? load_gamma_shifted(gamma, (t + i * tpr) * E - shift, cols) : make_uint4(0, 0, 0, 0), f);
        else
            unpack_vec<T>(has(i) ? __ldg(reinterpret_cast<const uint4 *>(gamma) + t + i * tpr) : make_uint4(0, 0, 0, 0), f);
#pragma unroll
        for (int j = 0; j < H; ++j) out[j] = make_float2(f[2 * j], f[2 * j + 1]);
    };
    if constexpr (kKeepGamma) {
#pragma unroll
        for (int i = 0; i < VPT; ++i) load_gamma(i, g[i]);
    }
    uint4 v[VPT];
    auto load_row = [&](int64_t row) {
        if constexpr (SHIFTED) {
            const T *src = x + row * ld_x;
            const int s = dq::row_shift(src);
#pragma unroll
            for (int i = 0; i < VPT; ++i) v[i] = row < rows ? dq::load8_edge(src, (t + i * tpr) * E - s, cols) : make_uint4(0, 0, 0, 0);
        } else {
            const uint4 *src = reinterpret_cast<const uint4 *>(x + row * ld_x);
#pragma unroll
            for (int i = 0; i < VPT; ++i) v[i] = row < rows && has(i) ? __ldg(src + t + i * tpr) : make_uint4(0, 0, 0, 0);
        }
    };
    const int64_t step = static_cast<int64_t>(gridDim.x) * rows_per_cta;
    load_row(row);
    int parity = 0;
    // all rows of a CTA advance together (the barriers below); rows beyond the last one are zeros and write nothing
    for (int64_t base = static_cast<int64_t>(blockIdx.x) * rows_per_cta; base < rows; base += step, row += step, parity ^= 1) {
        set_shift(row);
        float2 f[VPT][H];
        float sumsq = 0.0f;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            float e[E];
            unpack_vec<T>(v[i], e);
#pragma unroll
            for (int j = 0; j < H; ++j) {
                f[i][j] = make_float2(e[2 * j], e[2 * j + 1]);
                sumsq = fmaf(e[2 * j], e[2 * j], sumsq);
                sumsq = fmaf(e[2 * j + 1], e[2 * j + 1], sumsq);
            }
        }
        load_row(row + step);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sumsq += __shfl_xor_sync(0xffffffffu, sumsq, o);
        if (tpr > 32) {
            if (lane == 0) s_part[parity][0][warp] = sumsq;
            __syncthreads();
            float s = 0.0f;
            for (int w = 0; w < warps_per_row; ++w) s += s_part[parity][0][w0 + w];
            sumsq = s;
        }
        const float rstd = rstd_of(sumsq, cols, eps);
        const bool row_ok = row < rows;
        if (row_ok && t == 0) rstd_out[row] = rstd;

        // y = (x * rstd) * gamma, rounded once to T
        const float2 rstd2 = make_float2(rstd, rstd);
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            float2 gi[H];
            if constexpr (!kKeepGamma) load_gamma(i, gi);
            float e[E];
#pragma unroll
            for (int j = 0; j < H; ++j) {
                const float2 n = mul2(mul2(f[i][j], rstd2), kKeepGamma ? g[kKeepGamma ? i : 0][j] : gi[j]);
                e[2 * j] = n.x;
                e[2 * j + 1] = n.y;
            }
            const uint4 w = pack_vec<T>(e);
            // guarded vectors hold zeros unless rstd is infinite or NaN: those rows are not finite anyway
            if (FULL || has(i)) amax = max_nan(amax, dq::absmax8<T>(w));  // of the rounded values
            unpack_vec<T>(w, e);
#pragma unroll
            for (int j = 0; j < H; ++j) f[i][j] = make_float2(e[2 * j], e[2 * j + 1]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (tpr > 32) {
            if (lane == 0) s_part[parity][1][warp] = amax;
            __syncthreads();
            float m = 0.0f;
            for (int w = 0; w < warps_per_row; ++w) m = max_nan(m, s_part[parity][1][w0 + w]);
            amax = m;
        }
        const dq::RowQuant rq = dq::make_row_quant(amax);
        if (row_ok && t == 0) scale[row] = rq.scale;
        int8_t *dst = q + row * ld_q;
        auto store = [&](int i, const uint2 &b) {
            if constexpr (SHIFTED)
                dq::store8_edge(dst, (t + i * tpr) * E - shift, cols, b);
            else
                reinterpret_cast<uint2 *>(dst)[t + i * tpr] = b;
        };
        if (!rq.exact_only && rq.scale != 0.0f) {  // as dq::quantize8, two elements an instruction
            const float2 inv2 = make_float2(rq.inv, rq.inv), neg2 = make_float2(-rq.scale, -rq.scale);
            const float2 magic2 = make_float2(12582912.0f, 12582912.0f);
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                uint32_t b[E];
#pragma unroll
                for (int j = 0; j < H; ++j) {
                    const float2 q0 = mul2(f[i][j], inv2);
                    const float2 r = add2(fma2(fma2(q0, neg2, f[i][j]), inv2, q0), magic2);
                    b[2 * j] = __float_as_uint(r.x);
                    b[2 * j + 1] = __float_as_uint(r.y);
                }
                if (row_ok && has(i)) store(i, dq::gather_low_bytes(b));
            }
        } else if (row_ok) {
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                float e[E];
#pragma unroll
                for (int j = 0; j < H; ++j) {
                    e[2 * j] = f[i][j].x;
                    e[2 * j + 1] = f[i][j].y;
                }
                if (has(i)) store(i, dq::quantize8(e, rq, false));
            }
        }
    }
}

// Any column count, stride or alignment: one CTA per row, the row is read again from L2 for each pass.
// Its successor is released at its end, as dynamic_quant_generic_kernel's is and for its reason (fused, 300 x 16383, back
// to back: 32.5 -> 23.4 us; 25.1 without an overlapped launch).
template <typename T, bool QUANT>
__global__ void __launch_bounds__(256)
rms_norm_generic_kernel(const T *__restrict__ x, int64_t rows, int64_t cols, int64_t ld_x, const T *__restrict__ gamma,
                        float eps, T *__restrict__ y, int64_t ld_y, int8_t *__restrict__ q, int64_t ld_q,
                        float *__restrict__ scale, float *__restrict__ rstd_out) {
    pdl_wait();
    __shared__ float s_part[8];
    __shared__ float s_bcast;
    const int64_t row = blockIdx.x;
    const T *src = x + row * ld_x;
    float sumsq = 0.0f;
    for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
        const float f = to_float(src[c]);
        sumsq = fmaf(f, f, sumsq);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sumsq += __shfl_xor_sync(0xffffffffu, sumsq, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = sumsq;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.0f;
        for (int w = 0; w < 8; ++w) s += s_part[w];
        s_bcast = rstd_of(s, static_cast<int>(cols), eps);
        rstd_out[row] = s_bcast;
    }
    __syncthreads();
    const float rstd = s_bcast;
    auto y_of = [&](int64_t c) {
        return to_float(from_float<T>(__fmul_rn(__fmul_rn(to_float(src[c]), rstd), to_float(gamma[c]))));
    };
    if constexpr (!QUANT) {
        for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) y[row * ld_y + c] = from_float<T>(y_of(c));
    } else {
        float amax = 0.0f;
        for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) amax = max_nan(amax, fabsf(y_of(c)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        __syncthreads();
        if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = amax;
        __syncthreads();
        float m = 0.0f;
        for (int w = 0; w < 8; ++w) m = max_nan(m, s_part[w]);
        const dq::RowQuant rq = dq::make_row_quant(m);
        if (threadIdx.x == 0) scale[row] = rq.scale;
        for (int64_t c = threadIdx.x; c < cols; c += blockDim.x)
            q[row * ld_q + c] = static_cast<int8_t>(dq::quant_one(y_of(c), rq));
    }
}

template <typename T, bool QUANT>
int launch_rms_norm(const T *x, int64_t rows, int64_t cols, int64_t ld_x, const T *gamma, float eps, T *y, int64_t ld_y,
                    int8_t *q, int64_t ld_q, float *scale, float *rstd, cudaStream_t stream) {
    constexpr int E = VecOf<T>::kElems;
    const bool out_ok = QUANT ? ((ld_q % 8 == 0) && (reinterpret_cast<uintptr_t>(q) & 7) == 0)
                              : ((ld_y % E == 0) && (reinterpret_cast<uintptr_t>(y) & 15) == 0);
    const bool vec_ok = (cols % E == 0) && (ld_x % E == 0) && out_ok && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                        (reinterpret_cast<uintptr_t>(gamma) & 15) == 0 && cols / E <= 512 * 8;
    // off the vector grid, but input and output by as much (16-bit types)
    bool shifted = false;
    if constexpr (E == 8) {
        shifted = !vec_ok && (reinterpret_cast<uintptr_t>(gamma) & 15) == 0 && cols + 7 <= 512 * 8 * E &&
                  (QUANT ? dq::same_shift(x, ld_x, 2, q, ld_q, 1) : dq::same_shift(x, ld_x, 2, y, ld_y, 2));
    }
    if (vec_ok || shifted) {
        const int nvec = static_cast<int>((shifted ? cols + 2 * E - 2 : cols) / E);
        int tpr = 32;
        // eight vectors per thread where the row is long enough: the kernels are bound by instruction issue, and
        // the per-thread fixed cost (row scale, reductions, index arithmetic) is then spread over more elements
        while (tpr < 512 && tpr * 8 < nvec) tpr <<= 1;
        const int need = (nvec + tpr - 1) / tpr;
        const int threads = tpr > 128 ? tpr : 128;  // small CTAs: the tail of the grid is one CTA long
        const int rows_per_cta = threads / tpr;
        const int64_t grid = (rows + rows_per_cta - 1) / rows_per_cta;
        const int icols = static_cast<int>(cols);
        if constexpr (QUANT) {
            if (tpr <= 256) {
                const bool full = nvec == tpr * need;
                auto pick = [&](auto v) {
                    constexpr int V = decltype(v)::value;
                    return shifted ? rms_norm_quant_walk_kernel<T, V, false, true>
                           : full  ? rms_norm_quant_walk_kernel<T, V, true> : rms_norm_quant_walk_kernel<T, V, false>;
                };
                using Kernel = decltype(&rms_norm_quant_walk_kernel<T, 1, true>);
                const Kernel kernels[8] = {pick(std::integral_constant<int, 1>()), pick(std::integral_constant<int, 2>()),
                                           pick(std::integral_constant<int, 3>()), pick(std::integral_constant<int, 4>()),
                                           pick(std::integral_constant<int, 5>()), pick(std::integral_constant<int, 6>()),
                                           pick(std::integral_constant<int, 7>()), pick(std::integral_constant<int, 8>())};
                const int64_t resident = static_cast<int64_t>(sm_count()) * (512 / threads);
                QMM_CUDA_OK(launch_pdl(kernels[need - 1], dim3(static_cast<unsigned>(grid < resident ? grid : resident)),
                                       dim3(static_cast<unsigned>(threads)), 0, stream, x, rows, icols, ld_x, gamma, eps, q, ld_q,
                                       scale, rstd, tpr));
                return QMM_OK;
            }
        }
        auto kern = rms_norm_vec_kernel<T, 8, QUANT>;  // fused: rows of more than 256 x 8 vectors only
        if constexpr (!QUANT) {
            if (need <= 1) kern = rms_norm_vec_kernel<T, 1, QUANT>;
            else if (need <= 2) kern = rms_norm_vec_kernel<T, 2, QUANT>;
            else if (need <= 4) kern = rms_norm_vec_kernel<T, 4, QUANT>;
        }
        if constexpr (E == 8 && QUANT) {
            if (shifted) kern = rms_norm_vec_kernel<T, 8, QUANT, true>;
        } else if constexpr (E == 8) {
            if (shifted) {
                const decltype(kern) kernels[8] = {rms_norm_vec_kernel<T, 1, QUANT, true>, rms_norm_vec_kernel<T, 2, QUANT, true>,
                                                   rms_norm_vec_kernel<T, 3, QUANT, true>, rms_norm_vec_kernel<T, 4, QUANT, true>,
                                                   rms_norm_vec_kernel<T, 5, QUANT, true>, rms_norm_vec_kernel<T, 6, QUANT, true>,
                                                   rms_norm_vec_kernel<T, 7, QUANT, true>, rms_norm_vec_kernel<T, 8, QUANT, true>};
                kern = kernels[need - 1];
            }
        }
        QMM_CUDA_OK(launch_pdl(kern, dim3(static_cast<unsigned>(grid)), dim3(static_cast<unsigned>(threads)), 0, stream, x, rows,
                               icols, ld_x, gamma, eps, y, ld_y, q, ld_q, scale, rstd, tpr));
    } else {
        QMM_CUDA_OK(launch_pdl(rms_norm_generic_kernel<T, QUANT>, dim3(static_cast<unsigned>(rows)), dim3(256), 0, stream, x,
                               rows, cols, ld_x, gamma, eps, y, ld_y, q, ld_q, scale, rstd));
    }
    return QMM_OK;
}

}  // namespace
}  // namespace qmm

extern "C" int qmm_rms_norm(const void *x, int x_dtype, int64_t rows, int64_t cols, int64_t ld_x, const void *gamma,
                            double epsilon, void *y, int64_t ld_y, float *rstd, void *stream) {
    using namespace qmm;
    QMM_REQUIRE(rows >= 0 && cols > 0, "qmm_rms_norm: rows must be non-negative and cols positive");
    if (rows == 0) return QMM_OK;
    QMM_REQUIRE(x != nullptr && gamma != nullptr && y != nullptr && rstd != nullptr, "qmm_rms_norm: NULL operand");
    QMM_REQUIRE(ld_x >= cols && ld_y >= cols, "qmm_rms_norm: row stride smaller than the row length");
    QMM_REQUIRE(rows < (1ll << 31), "qmm_rms_norm: more than 2^31-1 rows");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const float eps = static_cast<float>(epsilon);
    switch (x_dtype) {
        case QMM_DTYPE_BF16:
            return launch_rms_norm<__nv_bfloat16, false>(static_cast<const __nv_bfloat16 *>(x), rows, cols, ld_x,
                                                         static_cast<const __nv_bfloat16 *>(gamma), eps,
                                                         static_cast<__nv_bfloat16 *>(y), ld_y, nullptr, 0, nullptr, rstd, s);
        case QMM_DTYPE_F16:
            return launch_rms_norm<__half, false>(static_cast<const __half *>(x), rows, cols, ld_x,
                                                  static_cast<const __half *>(gamma), eps, static_cast<__half *>(y), ld_y,
                                                  nullptr, 0, nullptr, rstd, s);
        case QMM_DTYPE_F32:
            return launch_rms_norm<float, false>(static_cast<const float *>(x), rows, cols, ld_x,
                                                 static_cast<const float *>(gamma), eps, static_cast<float *>(y), ld_y,
                                                 nullptr, 0, nullptr, rstd, s);
        default:
            return fail(QMM_ERR_UNSUPPORTED, "qmm_rms_norm: dtype must be bf16, f16 or f32");
    }
}

extern "C" int qmm_rms_norm_dynamic_quant(const void *x, int x_dtype, int64_t rows, int64_t cols, int64_t ld_x,
                                          const void *gamma, double epsilon, int8_t *q, int64_t ld_q, float *scale,
                                          float *rstd, void *stream) {
    using namespace qmm;
    QMM_REQUIRE(rows >= 0 && cols > 0, "qmm_rms_norm_dynamic_quant: rows must be non-negative and cols positive");
    if (rows == 0) return QMM_OK;
    QMM_REQUIRE(x != nullptr && gamma != nullptr && q != nullptr && scale != nullptr && rstd != nullptr,
                "qmm_rms_norm_dynamic_quant: NULL operand");
    QMM_REQUIRE(ld_x >= cols && ld_q >= cols, "qmm_rms_norm_dynamic_quant: row stride smaller than the row length");
    QMM_REQUIRE(rows < (1ll << 31), "qmm_rms_norm_dynamic_quant: more than 2^31-1 rows");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const float eps = static_cast<float>(epsilon);
    switch (x_dtype) {
        case QMM_DTYPE_BF16:
            return launch_rms_norm<__nv_bfloat16, true>(static_cast<const __nv_bfloat16 *>(x), rows, cols, ld_x,
                                                        static_cast<const __nv_bfloat16 *>(gamma), eps, nullptr, 0, q, ld_q,
                                                        scale, rstd, s);
        case QMM_DTYPE_F16:
            return launch_rms_norm<__half, true>(static_cast<const __half *>(x), rows, cols, ld_x,
                                                 static_cast<const __half *>(gamma), eps, nullptr, 0, q, ld_q, scale, rstd,
                                                 s);
        default:
            return fail(QMM_ERR_UNSUPPORTED, "qmm_rms_norm_dynamic_quant: dtype must be bf16 or f16");
    }
}
