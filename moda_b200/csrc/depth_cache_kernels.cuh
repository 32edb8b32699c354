// In-place depth-KV cache: one layer's K and V rows are copied into their slot of a persistent
// [B, T, Lmax, H, D] cache, which later layers read as depth K/V through Params::Ls.  Replaces the
// reference caller's per-layer rebuild of the whole cache (torch.stack over all earlier layers,
// reshape, contiguous: vision_tasks/deit/models.py:361-375), whose copies grow with the square of
// the layer count; here every K/V row is copied once.  The gradients of a slot come back out of a
// gradient cache of the same layout the same way.
#pragma once
#include "common.cuh"

namespace moda {
namespace cache {

// One thread per 16-byte chunk of a (b, t, h) row of k and of v.  chunks = D / 8.  kTake: from the
// slot of the caches ck, cv to k, v; otherwise from k, v into the slot.
template <int kChunks, bool kTake>
__global__ void __launch_bounds__(256) slot_kernel(View k, View v, View ck, View cv, int B, int T, int H, int Ls, int slot) {
  const int64_t n = (int64_t)B * T * H * kChunks;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % kChunks);
    int64_t r = i / kChunks;
    const int h = (int)(r % H); r /= H;
    const int t = (int)(r % T);
    const int b = (int)(r / T);
    const int64_t cache_row = (int64_t)t * Ls + slot;
    auto at = [&](const View& x, int64_t row) { return reinterpret_cast<uint4*>(static_cast<unsigned char*>(x.ptr) + 2 * (x.off(b, row, h) + c * 8)); };
    uint4 *k4 = at(k, t), *v4 = at(v, t), *ck4 = at(ck, cache_row), *cv4 = at(cv, cache_row);
    const uint4 x = kTake ? *ck4 : *k4, y = kTake ? *cv4 : *v4;
    *(kTake ? k4 : ck4) = x;
    *(kTake ? v4 : cv4) = y;
  }
}

}  // namespace cache
}  // namespace moda
