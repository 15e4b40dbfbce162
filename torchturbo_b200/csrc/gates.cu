// Gates whose fp32 values stand in for fp32 torch operations: exponentials, divisions and roots at full precision (the build
// compiles this source without --use_fast_math).
#include "common.cuh"
#include "rowops.cuh"

namespace ttb {

// ============================================================================
// Gated RMSNorm of short rows (head widths of the linear-attention layers): y = bf16(n * act(gate)) with
// n = bf16(bf16(x * rstd) * w), H = 8 L channels held by L lanes, so a warp normalises 32 / L rows with shuffles only.
//   dn = bf16(dy * act(gate)), dgate = dy * n * act'(gate), dx and dw as in the plain norm with dn in the place of dy
// Every rounding of the separate kernels (norm, fp32 product, cast) is kept.  A thread has its next row's loads under way while it works on
// one: 131072 rows of 128 (100 and 168 MB) from cold caches 37 -> 35 us forward and 62 -> 52 us backward with its column sums (memory
// alone: 16 and 27).  What is left over that is exponentials and divisions at full precision (approximate ones saved 6 and 10 us).
// ============================================================================
template <int L>
__device__ __forceinline__ float lane_group_sum(float v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// eight values of a row that is still on its way: the load stays here, the unpacking where the row is used
__device__ __forceinline__ uint4 load_here(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16(v)); }

template <int L>
__global__ void __launch_bounds__(256) gated_rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gate,
                                                               const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                                               float* __restrict__ rstd_out, long long R, float eps, int silu) {
  constexpr int H = 8 * L, ROWS = 256 / L;
  const int l = threadIdx.x % L, c = l * 8;
  float wf[8];
  load8(w + c, wf);
  // all lanes of a warp stay in the loop (the shuffles name the whole warp); rows past the end are computed and dropped
  const long long last = (R + ROWS - 1) / ROWS * ROWS;
  const long long step = static_cast<long long>(gridDim.x) * ROWS;
  long long row = static_cast<long long>(blockIdx.x) * ROWS + threadIdx.x / L;
  uint4 nx, ng;
  auto fetch = [&](long long r) {      // (a row past the end is loaded as the last one)
    const long long at = (r < R ? r : R - 1) * H + c;
    nx = load_here(x + at); ng = load_here(gate + at);
  };
  fetch(row);
  for (; row < last; row += step) {
    const bool ok = row < R;
    const uint4 cx = nx, cg = ng;
    if (row + step < last) fetch(row + step);
    float f[8], g[8];
    unpack8(cx, f); unpack8(cg, g);
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    const float rstd = rsqrtf(lane_group_sum<L>(ss) / static_cast<float>(H) + eps);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      f[j] = round_bf16(round_bf16(f[j] * rstd) * wf[j]) * ((silu ? g[j] : 1.f) / (1.f + expf(-g[j])));
    }
    if (ok) {
      store8(y + row * H + c, f);
      if (l == 0) rstd_out[row] = rstd;
    }
  }
}

template <int L>
__global__ void __launch_bounds__(256) gated_rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                               const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ w,
                                                               const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                                                               __nv_bfloat16* __restrict__ dgate, float* __restrict__ dw_partial,
                                                               long long R, int silu) {
  constexpr int H = 8 * L, ROWS = 256 / L;
  __shared__ float red[ROWS][H];
  const int l = threadIdx.x % L, c = l * 8, r0 = threadIdx.x / L;
  float wf[8], dw[8] = {};
  load8(w + c, wf);
  const long long last = (R + ROWS - 1) / ROWS * ROWS;
  const long long step = static_cast<long long>(gridDim.x) * ROWS;
  long long row = static_cast<long long>(blockIdx.x) * ROWS + r0;
  uint4 nx, ng, nd;
  float nr;
  auto fetch = [&](long long r) {
    const long long k = r < R ? r : R - 1, at = k * H + c;
    nx = load_here(x + at); ng = load_here(gate + at); nd = load_here(dy + at);
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(nr) : "l"(rstd_in + k));
  };
  fetch(row);
  for (; row < last; row += step) {
    const bool ok = row < R;
    const uint4 cx = nx, cg = ng, cd = nd;
    const float rstd = nr;
    if (row + step < last) fetch(row + step);
    float f[8], g[8], d[8];
    unpack8(cx, f); unpack8(cg, g); unpack8(cd, d);
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sg = 1.f / (1.f + expf(-g[j])), act = silu ? g[j] * sg : sg;
      const float n = round_bf16(round_bf16(f[j] * rstd) * wf[j]);
      const float slope = silu ? sg * (1.f + g[j] * (1.f - sg)) : sg * (1.f - sg);
      g[j] = d[j] * n * slope;
      f[j] *= rstd;
      const float dn = round_bf16(d[j] * act);
      if (ok) dw[j] += dn * f[j];
      d[j] = dn * wf[j];
      dot += d[j] * f[j];
    }
    dot = lane_group_sum<L>(dot) / static_cast<float>(H);
#pragma unroll
    for (int j = 0; j < 8; ++j) d[j] = rstd * (d[j] - f[j] * dot);
    if (ok) {
      store8(dx + row * H + c, d);
      store8(dgate + row * H + c, g);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) red[r0][c + j] = dw[j];
  __syncthreads();
  for (int e = threadIdx.x; e < H; e += 256) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) s += red[r][e];
    dw_partial[static_cast<long long>(blockIdx.x) * H + e] = s;
  }
}

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

// ============================================================================
// Gates of a gated delta net, per head, from the two raw projections (bf16 [rows, H], any row stride):
//   g = -exp(A_h) softplus(a + dt_h),   beta = sigmoid(b),   fp32 [rows, H]
// The backward returns da and db and the sums behind d(A) and d(dt).  131,000 elements for 4096 tokens and 32 heads are no work for the
// chip: what counts is the number of launches, one forward and two backward here, ten and fifteen in torch (4096 x 32: 47 -> 4 us and
// 65 -> 9 us with their gaps).  The same fp32 functions as torch's, softplus the identity above 20.
// ============================================================================
__global__ void __launch_bounds__(256)
gdn_gate_fwd_kernel(const __nv_bfloat16* __restrict__ a, long long a_t, const __nv_bfloat16* __restrict__ b, long long b_t,
                    const void* __restrict__ A, int a_bf16, const void* __restrict__ dt, int dt_bf16, float* __restrict__ g,
                    float* __restrict__ beta, long long rows, int H) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= rows * H) return;
  const long long r = idx / H;
  const int h = static_cast<int>(idx - r * H);
  const float x = __bfloat162float(a[r * a_t + h]) + load_scalar(dt, h, dt_bf16), y = __bfloat162float(b[r * b_t + h]);
  g[idx] = -expf(load_scalar(A, h, a_bf16)) * (x > 20.f ? x : log1pf(expf(x)));
  beta[idx] = 1.f / (1.f + expf(-y));
}

// 32 heads and a share of the rows per block; part: fp32 [blocks, 2, H], d(A) then d(dt)
__global__ void __launch_bounds__(256)
gdn_gate_bwd_kernel(const float* __restrict__ dg, const float* __restrict__ dbeta, const __nv_bfloat16* __restrict__ a, long long a_t,
                    const void* __restrict__ A, int a_bf16, const void* __restrict__ dt, int dt_bf16, const float* __restrict__ beta,
                    __nv_bfloat16* __restrict__ da, __nv_bfloat16* __restrict__ db, float* __restrict__ part, long long rows, int H) {
  __shared__ float red[2][8][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, h = blockIdx.x * 32 + x;
  float sum_a = 0.f, sum_dt = 0.f;
  if (h < H) {
    const float e = expf(load_scalar(A, h, a_bf16)), t = load_scalar(dt, h, dt_bf16);
    for (long long r = static_cast<long long>(blockIdx.y) * 8 + y; r < rows; r += static_cast<long long>(gridDim.y) * 8) {
      const float z = __bfloat162float(a[r * a_t + h]) + t, d = dg[r * H + h], s = beta[r * H + h], ez = expf(z);
      const bool linear = z > 20.f;
      const float dz = -d * e * (linear ? 1.f : ez / (ez + 1.f));
      sum_a += -d * e * (linear ? z : log1pf(ez));
      sum_dt += dz;
      da[r * H + h] = __float2bfloat16(dz);
      db[r * H + h] = __float2bfloat16(dbeta[r * H + h] * (1.f - s) * s);
    }
  }
  red[0][y][x] = sum_a;
  red[1][y][x] = sum_dt;
  __syncthreads();
  if (y < 2 && h < H) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += red[y][i][x];
    part[(static_cast<long long>(blockIdx.y) * 2 + y) * H + h] = s;
  }
}

}  // namespace ttb

using namespace ttb;

#define STREAM(s) reinterpret_cast<cudaStream_t>(s)
#define LAUNCH_RET() do { cudaError_t e__ = cudaGetLastError(); return e__ == cudaSuccess ? 0 : 400 + (int)e__; } while (0)

// H: 64, 128 or 256; all bf16 pointers on 16-byte boundaries
TTB_EXPORT int ttb_gated_rmsnorm_fwd(const void* x, const void* gate, const void* w, void* y, float* rstd, long long R, int H, float eps,
                                     int silu, int grid, void* stream) {
  if (R == 0) return 0;
  if (((uintptr_t)x | (uintptr_t)gate | (uintptr_t)w | (uintptr_t)y) & 15) return 902;
  auto X = (const __nv_bfloat16*)x; auto G = (const __nv_bfloat16*)gate; auto W = (const __nv_bfloat16*)w;
  auto Y = (__nv_bfloat16*)y;
  if (H == 64) gated_rmsnorm_fwd_kernel<8><<<grid, 256, 0, STREAM(stream)>>>(X, G, W, Y, rstd, R, eps, silu);
  else if (H == 128) gated_rmsnorm_fwd_kernel<16><<<grid, 256, 0, STREAM(stream)>>>(X, G, W, Y, rstd, R, eps, silu);
  else if (H == 256) gated_rmsnorm_fwd_kernel<32><<<grid, 256, 0, STREAM(stream)>>>(X, G, W, Y, rstd, R, eps, silu);
  else return 901;
  LAUNCH_RET();
}

// dw_partial must hold grid * H floats
TTB_EXPORT int ttb_gated_rmsnorm_bwd(const void* dy, const void* x, const void* gate, const void* w, const float* rstd, void* dx,
                                     void* dgate, float* dw_partial, void* dw_out, long long R, int H, int silu, int grid, void* stream) {
  if (R == 0) return 0;
  if (((uintptr_t)dy | (uintptr_t)x | (uintptr_t)gate | (uintptr_t)w | (uintptr_t)dx | (uintptr_t)dgate) & 15) return 902;
  auto D = (const __nv_bfloat16*)dy; auto X = (const __nv_bfloat16*)x; auto G = (const __nv_bfloat16*)gate;
  auto W = (const __nv_bfloat16*)w; auto DX = (__nv_bfloat16*)dx; auto DG = (__nv_bfloat16*)dgate;
  if (H == 64) gated_rmsnorm_bwd_kernel<8><<<grid, 256, 0, STREAM(stream)>>>(D, X, G, W, rstd, DX, DG, dw_partial, R, silu);
  else if (H == 128) gated_rmsnorm_bwd_kernel<16><<<grid, 256, 0, STREAM(stream)>>>(D, X, G, W, rstd, DX, DG, dw_partial, R, silu);
  else if (H == 256) gated_rmsnorm_bwd_kernel<32><<<grid, 256, 0, STREAM(stream)>>>(D, X, G, W, rstd, DX, DG, dw_partial, R, silu);
  else return 901;
  colsum(dw_partial, dw_out, 1, grid, H, STREAM(stream));
  LAUNCH_RET();
}

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

// a, b: bf16 [rows, H] with row strides a_t, b_t; A, dt: [H] fp32 or bf16; g, beta: fp32 [rows, H]
TTB_EXPORT int ttb_gdn_gate_fwd(const void* a, long long a_t, const void* b, long long b_t, const void* A, int a_bf16, const void* dt, int dt_bf16,
                                float* g, float* beta, long long rows, int H, void* stream) {
  const long long n = rows * H;
  if (n == 0) return 0;
  gdn_gate_fwd_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, STREAM(stream)>>>((const __nv_bfloat16*)a, a_t, (const __nv_bfloat16*)b, b_t, A,
                                                                                       a_bf16, dt, dt_bf16, g, beta, rows, H);
  LAUNCH_RET();
}

// da, db: bf16 [rows, H] contiguous; part: fp32 [blocks, 2, H]; sums: [2, H] (d(A), d(dt)), fp32 or bf16
TTB_EXPORT int ttb_gdn_gate_bwd(const float* dg, const float* dbeta, const void* a, long long a_t, const void* A, int a_bf16, const void* dt,
                                int dt_bf16, const float* beta, void* da, void* db, float* part, void* sums, int out_bf16, long long rows, int H,
                                int blocks, void* stream) {
  if (rows == 0 || H == 0) return 0;
  gdn_gate_bwd_kernel<<<dim3((H + 31) / 32, blocks), 256, 0, STREAM(stream)>>>(dg, dbeta, (const __nv_bfloat16*)a, a_t, A, a_bf16, dt, dt_bf16, beta,
                                                                             (__nv_bfloat16*)da, (__nv_bfloat16*)db, part, rows, H);
  colsum(part, sums, out_bf16, blocks, 2 * H, STREAM(stream));
  LAUNCH_RET();
}
