// readback.h -- large results from the GPU into the caller's (pageable) arrays.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <functional>

namespace lbgpu {

// Brings `items` items of `item_bytes` each back.  fill(k0, k1, dst) launches on `stream` the kernels that
// write items k0..k1-1 to dst, which is pinned host memory the GPU reaches; take(k0, k1, src) copies
// them from there into the caller's arrays.  Both are called from several threads at once for large
// results, for ranges that do not overlap.  Returns when everything has arrived, or the first CUDA
// error (nothing is in flight then either).
cudaError_t read_back(int device, cudaStream_t stream, long long items, size_t item_bytes,
                      const std::function<void(long long, long long, double *)> &fill,
                      const std::function<void(long long, long long, const double *)> &take);

// Gives back the pinned memory that is kept between calls (the last lattice went).
void read_back_release();

}  // namespace lbgpu
