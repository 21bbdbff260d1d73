// Prefix sums and stable compaction of lists of up to some millions of items.
#pragma once
#include <stdint.h>

#include "internal.hpp"

namespace eqtl {
namespace dev {

// Sum of v over the lower threads of a block (blockDim.x a multiple of 32, at
// most 1024); total = over all. sm: 33 values.
template <class T>
__device__ __forceinline__ T block_prefix(T v, T* sm, T& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  T s = v;
#pragma unroll
  for (int o = 1; o < 32; o *= 2) {
    const T x = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += x;
  }
  __syncthreads();  // sm of an earlier call has been read
  if (lane == 31) sm[w] = s;
  __syncthreads();
  if (w == 0) {
    const T x = lane < nw ? sm[lane] : T(0);
    T y = x;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const T z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    sm[lane] = y - x;
    if (lane == 31) sm[32] = y;
  }
  __syncthreads();
  total = sm[32];
  return sm[w] + s - v;
}

// Exclusive prefix sums of v in place, by one block of 1024; total (optional).
template <class T>
__global__ void __launch_bounds__(1024) prefix_kernel(T* __restrict__ v, int64_t n, T* total) {
  __shared__ T sm[33];
  T carry = 0;
  for (int64_t base = 0; base < n; base += 4096) {
    const int64_t i = base + 4 * threadIdx.x;
    T x[4], s = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x[j] = i + j < n ? v[i + j] : T(0);
      s += x[j];
    }
    T all, at = carry + block_prefix(s, sm, all);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i + j < n) v[i + j] = at;
      at += x[j];
    }
    carry += all;
  }
  if (total && threadIdx.x == 0) *total = carry;
}

// Stable compaction into two lists: f.test(i) is 1 in the low half for an entry
// of the first list, 1 in the high half for one of the second; f.emit(i, t, at)
// gets the places in both. Blocks of 1024 items.
constexpr int kCompactTile = 1024;
template <class F>
__global__ void __launch_bounds__(256) compact_count_kernel(F f, uint64_t* __restrict__ blk) {
  __shared__ uint64_t sm[33];
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kCompactTile + 4 * threadIdx.x, n = f.size();
  uint64_t s = 0, all;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (i + j < n) s += f.test(i + j);
  block_prefix(s, sm, all);
  if (threadIdx.x == 0) blk[blockIdx.x] = all;
}
template <class F>
__global__ void __launch_bounds__(256) compact_emit_kernel(F f, const uint64_t* __restrict__ blk) {
  __shared__ uint64_t sm[33];
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kCompactTile + 4 * threadIdx.x, n = f.size();
  uint64_t t[4], s = 0, all;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    t[j] = i + j < n ? f.test(i + j) : 0;
    s += t[j];
  }
  uint64_t at = blk[blockIdx.x] + block_prefix(s, sm, all);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (t[j]) f.emit(i + j, t[j], at);
    at += t[j];
  }
}

}  // namespace dev

inline unsigned blocks(int64_t n, int64_t per) {
  return static_cast<unsigned>(std::max<int64_t>((n + per - 1) / per, 1));
}

// f over its f.size() <= n_max items; *total (device) = the two lists' lengths.
template <class F>
void compact(eqtl_ctx* ctx, const F& f, int64_t n_max, uint64_t* total) {
  const unsigned nb = blocks(n_max, dev::kCompactTile);
  DevBuf<uint64_t>& blk = ctx->ws.res_blk;
  blk.alloc(nb);
  ctx->launches += 3;
  dev::compact_count_kernel<F><<<nb, 256, 0, ctx->stream>>>(f, blk.p);
  dev::prefix_kernel<uint64_t><<<1, 1024, 0, ctx->stream>>>(blk.p, nb, total);
  dev::compact_emit_kernel<F><<<nb, 256, 0, ctx->stream>>>(f, blk.p);
  EQTL_CUDA(cudaGetLastError());
}

}  // namespace eqtl
