// Gates whose fp32 values stand in for fp32 torch operations: exponentials, divisions and roots at full precision (the build
// compiles this source without --use_fast_math).
#include "common.cuh"
#include "rowops.cuh"

namespace ttb {

// ============================================================================
// Kimi delta attention gate: per-channel log decay of [rows, H, 128] from the raw projection,
//   d = -exp(A_h) softplus(x)   or, with a lower bound,   d = bound * sigmoid(exp(A_h) x),      x = g + dt
// One block row of 128 channels per head; the backward returns dg and, per block of rows, the channel sums behind d(dt) and
// d(A), which colsum adds up in a fixed order.  fp32 arithmetic; softplus is the identity above 20, as in torch.
// In torch this is about seven launches forward and fifteen backward over fp32 tensors; here it is one each way and a column sum
// (35 -> 21 launches for the operator); 2047 x 8 heads: 7 and 13 us (6 and 10 with approximate exponentials).
// ============================================================================
__device__ __forceinline__ float load_scalar(const void* p, long long i, int bf16) {
  return bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]) : reinterpret_cast<const float*>(p)[i];
}

__global__ void __launch_bounds__(128)
kda_gate_fwd_kernel(const __nv_bfloat16* __restrict__ g, const void* __restrict__ A, int a_bf16, const void* __restrict__ dt,
                    int dt_bf16, float* __restrict__ out, long long rows, int H, int bounded, float bound, int rows_per_block) {
  const int h = blockIdx.x;
  const long long col = static_cast<long long>(h) * 128 + threadIdx.x, step = static_cast<long long>(H) * 128;
  const float a = expf(load_scalar(A, h, a_bf16)), b = dt ? load_scalar(dt, col, dt_bf16) : 0.f;
  const long long r0 = static_cast<long long>(blockIdx.y) * rows_per_block, r1 = min(r0 + rows_per_block, rows);
#pragma unroll 4
  for (long long r = r0; r < r1; ++r) {
    const float x = __bfloat162float(g[r * step + col]) + b;
    out[r * step + col] = bounded ? bound / (1.f + expf(-a * x)) : -a * (x > 20.f ? x : log1pf(expf(x)));
  }
}

__global__ void __launch_bounds__(128)
kda_gate_bwd_kernel(const float* __restrict__ dd, const __nv_bfloat16* __restrict__ g, const void* __restrict__ A, int a_bf16,
                    const void* __restrict__ dt, int dt_bf16, __nv_bfloat16* __restrict__ dg, float* __restrict__ part,
                    long long rows, int H, int bounded, float bound, int rows_per_block) {
  const int h = blockIdx.x;
  const long long col = static_cast<long long>(h) * 128 + threadIdx.x, step = static_cast<long long>(H) * 128;
  const float a = expf(load_scalar(A, h, a_bf16)), b = dt ? load_scalar(dt, col, dt_bf16) : 0.f;
  const long long r0 = static_cast<long long>(blockIdx.y) * rows_per_block, r1 = min(r0 + rows_per_block, rows);
  float sum_dt = 0.f, sum_a = 0.f;
#pragma unroll 4
  for (long long r = r0; r < r1; ++r) {
    const float x = __bfloat162float(g[r * step + col]) + b, d = dd[r * step + col];
    float dx, da;
    if (bounded) {
      const float sg = 1.f / (1.f + expf(-a * x)), slope = d * bound * sg * (1.f - sg);
      dx = slope * a;
      da = slope * a * x;
    } else {
      const bool linear = x > 20.f;
      const float e = expf(x);
      dx = -d * a * (linear ? 1.f : e / (1.f + e));
      da = -d * a * (linear ? x : log1pf(e));
    }
    dg[r * step + col] = __float2bfloat16(dx);
    sum_dt += dx;
    sum_a += da;
  }
  part[blockIdx.y * 2 * step + col] = sum_dt;
  part[(blockIdx.y * 2 + 1) * step + col] = sum_a;
}

}  // namespace ttb

using namespace ttb;

#define STREAM(s) reinterpret_cast<cudaStream_t>(s)
#define LAUNCH_RET() do { cudaError_t e__ = cudaGetLastError(); return e__ == cudaSuccess ? 0 : 400 + (int)e__; } while (0)

static int kda_gate_rows(long long rows, int H, int& blocks) {
  if (rows <= 0 || H <= 0) {
    blocks = 0;
    return 1;
  }
  long long want = (148LL * 8 + H - 1) / H;                 // about eight blocks per SM
  if (want > rows) want = rows;
  const int per = static_cast<int>((rows + want - 1) / want);
  blocks = static_cast<int>((rows + per - 1) / per);
  return per;
}

TTB_EXPORT int ttb_kda_gate_row_blocks(long long rows, int H) {
  int blocks = 0;
  kda_gate_rows(rows, H, blocks);
  return blocks;
}

TTB_EXPORT int ttb_kda_gate_fwd(const void* g, const void* A, int a_bf16, const void* dt, int dt_bf16, float* out, long long rows,
                                int H, int bounded, float bound, void* stream) {
  if (rows == 0 || H == 0) return 0;
  int blocks;
  const int per = kda_gate_rows(rows, H, blocks);
  kda_gate_fwd_kernel<<<dim3(H, blocks), 128, 0, STREAM(stream)>>>((const __nv_bfloat16*)g, A, a_bf16, dt, dt_bf16, out, rows, H,
                                                                  bounded, bound, per);
  LAUNCH_RET();
}

// part: fp32 [row_blocks, 2, H * 128]; sums: fp32 [2, H * 128] (d(dt), then the channel sums of d(A))
TTB_EXPORT int ttb_kda_gate_bwd(const float* dd, const void* g, const void* A, int a_bf16, const void* dt, int dt_bf16, void* dg,
                                float* part, float* sums, long long rows, int H, int bounded, float bound, void* stream) {
  if (rows == 0 || H == 0) return 0;
  int blocks;
  const int per = kda_gate_rows(rows, H, blocks);
  kda_gate_bwd_kernel<<<dim3(H, blocks), 128, 0, STREAM(stream)>>>(dd, (const __nv_bfloat16*)g, A, a_bf16, dt, dt_bf16,
                                                                  (__nv_bfloat16*)dg, part, rows, H, bounded, bound, per);
  colsum(part, sums, 0, blocks, 2 * H * 128, STREAM(stream));
  LAUNCH_RET();
}
