// Launchers of merkle_tensor.cu, called by merkle.cu's dispatch.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "kernels.h"

namespace whir {
namespace gpu {

cudaError_t init_poseidon2_tensor();  // per device: tables, attributes
// digests on a 16-byte boundary
void hash_rows_tensor(const uint32_t *rows, size_t n_rows, int row_len, uint32_t *digests,
                      cudaStream_t st, const WaitReport &report);
void compress_level_tensor(const uint32_t *src, uint32_t *dst, size_t half, cudaStream_t st,
                           const WaitReport &report);

}  // namespace gpu
}  // namespace whir
