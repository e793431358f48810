// Transposition of a batch of matrices, fp32.
#pragma once

#include <cuda_runtime.h>

namespace bc {
namespace gpu {

// out[b][c][r] = in[b][r][c]; the elements of a row are adjacent, `*_row` and `*_batch` are distances in elements.
cudaError_t transpose(const float* in, float* out, int batch, int rows, int cols, long long in_row, long long in_batch, long long out_row,
                      long long out_batch, cudaStream_t stream);

}  // namespace gpu
}  // namespace bc
