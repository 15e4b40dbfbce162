// Column sums shared by the kernels that reduce over rows.
#pragma once
#include "common.cuh"

namespace ttb {

// Column sum of partial[rows][H] -> out[H] (fp32 or bf16); deterministic order.  32 columns and 32 row groups per block:
// the sums are a few hundred rows long at most, so what counts is how many loads are in flight (2048 columns: 4.9 us with one
// thread per column, 2.3 now; the six sums of a ViT block 76 and 19 us).
__device__ __forceinline__ void store_scalar(float* p, float v) { *p = v; }
__device__ __forceinline__ void store_scalar(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }

template <typename Out>
static __global__ void __launch_bounds__(1024) colsum_kernel(const float* __restrict__ partial, Out* __restrict__ out, int rows, int H) {
  __shared__ float part[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + x;
  float s = 0.f;
  if (c < H) {
#pragma unroll 4
    for (int r = y; r < rows; r += 32) s += partial[static_cast<long long>(r) * H + c];
  }
  part[y][x] = s;
  __syncthreads();
  s = warp_sum(part[x][y]);
  if (x == 0 && blockIdx.x * 32 + y < H) store_scalar(out + blockIdx.x * 32 + y, s);
}
static void colsum(const float* partial, void* out, int out_bf16, int rows, int H, cudaStream_t st) {
  if (out_bf16) colsum_kernel<<<(H + 31) / 32, 1024, 0, st>>>(partial, static_cast<__nv_bfloat16*>(out), rows, H);
  else colsum_kernel<<<(H + 31) / 32, 1024, 0, st>>>(partial, static_cast<float*>(out), rows, H);
}

}  // namespace ttb
