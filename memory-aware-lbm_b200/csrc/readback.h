// readback.h -- large results from the GPU into the caller's (pageable) arrays.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace lbgpu {

// Brings `items` items of `item_bytes` each back.  fill(k0, k1, dst) launches on `stream` the kernels that
// write items k0..k1-1 to dst, which is pinned host memory the GPU reaches; take(k0, k1, src) copies
// them from there into the caller's arrays.  Both are called from several threads at once for large
// results, for ranges that do not overlap.  Returns when everything has arrived, or the first CUDA
// error (nothing is in flight then either).
// fill and take are functions or lambdas that outlive the call; nothing here allocates memory of the host's heap but
// for threads, without which it goes on.
template <class P>
struct RangeFn {
    const void *object;
    void (*call)(const void *, long long, long long, P *);
    template <class F>
    RangeFn(const F &f)
        : object(&f), call([](const void *o, long long a, long long b, P *p) { (*static_cast<const F *>(o))(a, b, p); })
    {
    }
    void operator()(long long a, long long b, P *p) const { call(object, a, b, p); }
};
cudaError_t read_back(int device, cudaStream_t stream, long long items, size_t item_bytes, RangeFn<double> fill,
                      RangeFn<const double> take);

// Gives back the pinned memory that is kept between calls (the last lattice went).
void read_back_release();

}  // namespace lbgpu
