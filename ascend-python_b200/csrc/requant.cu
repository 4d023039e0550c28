// int8 output of npu_quant_matmul (`output_dtype = int8`, with the optional `offset`).
//
// The reference does not define this operator's arithmetic; the stated choice here (x1, x2, scale, offset,
// pertoken_scale, bias, output_dtype) is:
//     acc[m,n] = sum_k x1[m,k] * x2[k,n] + bias[n]                      int32, exact (bias int32)
//     v        = float(acc) * scale[n] (* pertoken_scale[m]) (+ offset[n])   fp32, one rounding per operation
//     out      = clamp(rint(v), -128, 127)                              round half to even
// The requantization is one more output type of the matmul kernels' epilogue.  (As a pass of its own over an int32
// accumulator it cost 5 bytes of traffic per output element and a launch: 2048 x 14336 x 4096 took 118 us, now 98.)
#include "qmm_common.cuh"
#include "w8a8_epilogue.cuh"

namespace qmm {
int quant_matmul_dispatch(const int8_t *x1, int64_t ld_x1, const int8_t *x2, int64_t x2_sk, int64_t x2_sn,
                          const EpilogueParams &ep, int out_dtype, int64_t K, int algo, void *workspace,
                          size_t workspace_bytes, cudaStream_t stream, LaunchOptions *opts);
// whether the kernel that QMM_ALGO_AUTO takes shares sums through scratch
bool quant_matmul_wants_scratch(const int8_t *x1, int64_t ld_x1, const int8_t *x2, int64_t x2_sk, int64_t x2_sn, int64_t M,
                                int64_t N, int64_t K);
int validate_quant_matmul(const int8_t *x1, int64_t ld_x1, const int8_t *x2, int64_t x2_sk, int64_t x2_sn,
                          const float *scale, int64_t scale_len, const void *bias, int bias_dtype, void *out,
                          int out_dtype, int64_t ld_out, int64_t M, int64_t N, int64_t K);
namespace {
size_t align256(size_t v) { return (v + 255) / 256 * 256; }
}  // namespace
}  // namespace qmm

extern "C" int qmm_quant_matmul_workspace_size(int64_t M, int64_t N, int64_t K, int algo, size_t *bytes);

extern "C" int qmm_quant_matmul_int8_workspace_size(int64_t M, int64_t N, int64_t K, size_t *bytes) {
    using namespace qmm;
    QMM_REQUIRE(bytes != nullptr, "qmm_quant_matmul_int8_workspace_size: bytes is NULL");
    QMM_REQUIRE(M >= 0 && N >= 0 && K >= 0, "qmm_quant_matmul_int8_workspace_size: negative dimension");
    size_t inner = 0;
    int rc = qmm_quant_matmul_workspace_size(M, N, K, QMM_ALGO_AUTO, &inner);
    if (rc != QMM_OK) return rc;
    // the matmul's own scratch; never empty, so that a workspace is always asked for
    *bytes = inner > 0 ? align256(inner) : 256;
    return QMM_OK;
}

extern "C" int qmm_quant_matmul_int8(const int8_t *x1, int64_t ld_x1, const int8_t *x2, int64_t x2_stride_k,
                                     int64_t x2_stride_n, const float *scale, int64_t scale_len, const float *offset,
                                     int64_t offset_len, const float *pertoken_scale, const int32_t *bias, int8_t *out,
                                     int64_t ld_out, int64_t M, int64_t N, int64_t K, void *workspace,
                                     size_t workspace_bytes, void *stream) {
    using namespace qmm;
    QMM_REQUIRE(M >= 0 && N >= 0 && K >= 0, "qmm_quant_matmul_int8: negative dimension");
    if (M == 0 || N == 0) return QMM_OK;
    QMM_REQUIRE(out != nullptr && ld_out >= N, "qmm_quant_matmul_int8: out is NULL or ld_out smaller than N");
    QMM_REQUIRE(scale != nullptr && (scale_len == N || scale_len == 1), "qmm_quant_matmul_int8: scale must have N elements or one");
    QMM_REQUIRE(offset == nullptr || offset_len == N || offset_len == 1,
                "qmm_quant_matmul_int8: offset must have N elements or one");
    size_t need = 0, inner = 0;
    qmm_quant_matmul_int8_workspace_size(M, N, K, &need);
    qmm_quant_matmul_workspace_size(M, N, K, QMM_ALGO_AUTO, &inner);
    if (workspace == nullptr || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255) != 0)
        return fail(QMM_ERR_WORKSPACE, "qmm_quant_matmul_int8: workspace missing, not 256-byte aligned or smaller than "
                                       "qmm_quant_matmul_int8_workspace_size reports");
    // validated as the accumulator pass that the operator's definition names (int32 bias); K == 0 included
    int rc = validate_quant_matmul(x1, ld_x1, x2, x2_stride_k, x2_stride_n, nullptr, 0, bias, bias ? QMM_DTYPE_I32 : QMM_DTYPE_NONE,
                                   out, QMM_DTYPE_I32, ld_out, M, N, K);
    if (rc != QMM_OK) return rc;
    // the kernels that share sums through scratch want it zeroed; callers need not prepare it
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (inner > 0 && quant_matmul_wants_scratch(x1, ld_x1, x2, x2_stride_k, x2_stride_n, M, N, K)) QMM_CUDA_OK(cudaMemsetAsync(workspace, 0, inner, s));
    EpilogueParams ep;
    ep.scale = scale;
    ep.pertoken_scale = pertoken_scale;
    ep.bias = bias;
    ep.bias_dtype = bias ? QMM_DTYPE_I32 : QMM_DTYPE_NONE;
    ep.scale_is_scalar = (scale_len == 1 && N != 1) ? 1 : 0;
    ep.out = out;
    ep.ld_out = ld_out;
    ep.M = M;
    ep.N = N;
    ep.offset = offset;
    ep.offset_is_scalar = (offset_len == 1 && N != 1) ? 1 : 0;
    // K == 0: an empty reduction, the epilogue of zeros
    return quant_matmul_dispatch(x1, ld_x1, x2, x2_stride_k, x2_stride_n, ep, kOutI8, K, K == 0 ? QMM_ALGO_SIMT : QMM_ALGO_AUTO,
                                 inner ? workspace : nullptr, inner, s, nullptr);
}
