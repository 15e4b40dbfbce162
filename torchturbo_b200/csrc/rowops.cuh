// Loads of eight values and column sums, shared by the kernels that walk rows.
#pragma once
#include "common.cuh"

namespace ttb {

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}

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
