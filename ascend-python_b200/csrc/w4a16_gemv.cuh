// W4A16 matmul for one or two tokens over prepacked weights (w4a16_gemv.cu).
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <cuda_runtime.h>

namespace qmm {

constexpr int kGemvMaxM = 2;
// whether this kernel serves the call and is the faster one
bool prefer_gemv_tile(int64_t M, int64_t N, int64_t K);
// packed: the blocks of qmm_w4a16_prepack for this N and K
int launch_gemv_tile(const void *packed, const void *x, int x_dtype, int64_t ld_x, const void *bias, void *out, int64_t ld_out,
                     int64_t M, int64_t N, int64_t K, cudaStream_t stream);

}  // namespace qmm
