// Column sums of per-CTA partial weight gradients, fp32 [n_part, H] -> [H].
#pragma once
#include "common.cuh"

namespace rb {

// 32 columns a CTA (one 128-byte line per warp and row), the rows dealt over its 16 warps: H / 32 CTAs have a load per thread in flight
// where one thread per column walked all rows alone.  H = 4096, n_part = 592: 34 -> 4.5 us; the order of the sum is fixed.
template <typename T>
__global__ void __launch_bounds__(512) colsum_kernel(const float* __restrict__ partial, T* __restrict__ out, int n_part, int H) {
  __shared__ float part[16][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (c < H) {
#pragma unroll 4
    for (int p = warp; p < n_part; p += 16) acc += partial[(int64_t)p * H + c];
  }
  part[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && c < H) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 16; ++w) s += part[w][lane];
    out[c] = from_f<T>(s);
  }
}

template <typename T> void launch_colsum(const float* partial, void* out, int n_part, int H, cudaStream_t s) {
  colsum_kernel<T><<<RB_CEIL_DIV(H, 32), 512, 0, s>>>(partial, (T*)out, n_part, H);
}

}  // namespace rb
