// Bandwidth-bound training kernels for sm_100a: RMSNorm (+residual) fwd/bwd,
// fused QK-RMSNorm + rotary embedding fwd/bwd, SwiGLU fwd/bwd (with routing-prob
// scaling), cross-entropy with in-place gradient, multi-tensor AdamW with a
// device-side clip coefficient and multi-tensor squared-norm partials.
//
// Numerical contracts follow the reference's torch formulas:
//   RMSNorm   : fp32 x*rsqrt(mean(x^2)+eps) -> cast -> * weight        (ops/providers/native/rms_norm.py:16-22)
//   SwiGLU    : silu(gate) * up on [gate|up] halves, prob applied after the
//               activation                                             (ops/providers/native/swiglu.py:10-12,
//                                                                       models/modules/moe/experts.py:181-186)
//   CE        : fp32, reduction=sum, ignore_index=-100                (ops/providers/native/cross_entropy_loss.py:17-33)
//   AdamW     : torch fused AdamW math on fp32 shards                  (engine/backends/fsdp2/optimizers/adamw.py:226-251)
#include <type_traits>
#include "common.cuh"
#include "rowops.cuh"

namespace ttb {

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < nw) ? red[l] : 0.f;
  t = warp_sum(t);
  __syncthreads();
  return t;
}
// N sums in one exchange; red holds 32 N floats
template <int N>
__device__ __forceinline__ void block_sums(float (&v)[N], float* red) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = warp_sum(v[i]);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (l == 0) red[32 * i + w] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = l < nw ? red[32 * i + l] : 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = warp_sum(v[i]);
  __syncthreads();
}
// Launch of a row kernel whose blocks walk rows: eight columns a thread, so that a row is one load per operand and thread and the
// next row's loads fit into registers beside this one's.  Two rows at a time share their exchanges (two barriers and ten shuffles are half
// of a row's time) where every block has two and is small enough for two to run on an SM all the same (16384 x 4096 97 us with one row,
// 136 with two; 2850 x 1152 LayerNorm 18.3 and 16.5); blocks of more than 512 threads run one to an SM, and a second of them would only
// start when the first has ended (1000 x 8192 30 us with two, 23 with one).
static int row_threads(int cols) { return cols / 8 > 1024 ? 1024 : (cols / 8 + 31) / 32 * 32; }
// Blocks of one row each do not walk: what prepares a next row costs 0.15 us, of 3.0 (8 x 512) to 5.1 (61 x 2048).  Rows that leave an SM
// for each stay apart also where blocks are large (8 x 8192 10.3 us with two a block, 9.2 so).
struct RowPlan {
  int grid, threads;
  bool two, walk;
};
static RowPlan row_plan(long long rows, int cols, int grid) {
  RowPlan p{grid, row_threads(cols), false, false};
  if (p.threads > 512 && rows > device_sms()) p.grid = (grid + 1) / 2;
  if (p.threads <= 256 && rows > grid && rows < 2ll * grid) p.grid = static_cast<int>((rows + 1) / 2);
  if (p.grid > rows) p.grid = static_cast<int>(rows);
  p.two = p.threads <= 256 && rows > p.grid;
  p.walk = rows > p.grid;
  return p;
}
// the form of a row kernel that a plan asks for
#define ROW_KERNEL(name, plan) ((plan).two ? name<2, true> : (plan).walk ? name<1, true> : name<1, false>)
__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < nw) ? red[l] : -INFINITY;
  t = warp_max(t);
  __syncthreads();
  return t;
}

// ============================================================================
// RMSNorm forward.  y = bf16(bf16(x_sum * rstd) * w),  x_sum = x (+ residual).
// One block per row, 8 bf16 per thread per iteration (H % 8 == 0).
// ============================================================================
template <int MAX_ITERS>
__global__ void rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                   __nv_bfloat16* __restrict__ sum_out, float* __restrict__ rstd_out, int H, float eps,
                                   int one_plus_w) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * H;
  const __nv_bfloat16* rr = residual ? residual + row * H : nullptr;
  float vals[MAX_ITERS][8];
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int c = (it * blockDim.x + threadIdx.x) * 8;
    if (c >= H) break;
    uint4 u = *reinterpret_cast<const uint4*>(xr + c);
    float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), cc = unpack_bf16(u.z), d = unpack_bf16(u.w);
    float f[8] = {a.x, a.y, b.x, b.y, cc.x, cc.y, d.x, d.y};
    if (rr) {
      uint4 r = *reinterpret_cast<const uint4*>(rr + c);
      float2 ra = unpack_bf16(r.x), rb = unpack_bf16(r.y), rc = unpack_bf16(r.z), rd = unpack_bf16(r.w);
      float g[8] = {ra.x, ra.y, rb.x, rb.y, rc.x, rc.y, rd.x, rd.y};
      uint4 o;
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(__float2bfloat16(f[j] + g[j]));
      o.x = pack_bf16(f[0], f[1]); o.y = pack_bf16(f[2], f[3]); o.z = pack_bf16(f[4], f[5]); o.w = pack_bf16(f[6], f[7]);
      *reinterpret_cast<uint4*>(sum_out + row * H + c) = o;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      vals[it][j] = f[j];
      ss += f[j] * f[j];
    }
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / static_cast<float>(H) + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int c = (it * blockDim.x + threadIdx.x) * 8;
    if (c >= H) break;
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = vals[it][j];
    uint4 wu = *reinterpret_cast<const uint4*>(w + c);
    float2 wa = unpack_bf16(wu.x), wb = unpack_bf16(wu.y), wc = unpack_bf16(wu.z), wd = unpack_bf16(wu.w);
    float wf[8] = {wa.x, wa.y, wb.x, wb.y, wc.x, wc.y, wd.x, wd.y};
    float o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float xh = __bfloat162float(__float2bfloat16(f[j] * rstd));
      o[j] = xh * (one_plus_w ? 1.f + wf[j] : wf[j]);
    }
    uint4 ou;
    ou.x = pack_bf16(o[0], o[1]); ou.y = pack_bf16(o[2], o[3]); ou.z = pack_bf16(o[4], o[5]); ou.w = pack_bf16(o[6], o[7]);
    *reinterpret_cast<uint4*>(y + row * H + c) = ou;
  }
}

// RMSNorm backward.  Blocks walk rows, a thread owns eight columns; dw partials live in registers and are flushed to
// dw_partial[blockIdx.x][H] at the end.  The next row is on its way while this one is reduced: with its loads behind the
// reduction a row took two memory latencies.  With the column sum, before -> now: 16384 x 4096 189 -> 97 us (5.5 TB/s), 4096 x 8192
// 101 -> 59, 4096 x 2048 21 -> 19; LayerNorm 16384 x 4096 254 -> 107, 2850 x 1152 18.6 -> 16.5.
//   dx = rstd * (g - xhat * mean(g * xhat)),  g = dy * w,  xhat = x * rstd   (+ dres_in)
template <int ROWS, bool WALK>
__global__ void __launch_bounds__(ROWS == 1 ? 1024 : 256)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dres_in, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, long long T, int H, int one_plus_w) {
  __shared__ float red[32 * ROWS];
  const int c = threadIdx.x * 8;
  const bool mine = c < H;
  float dwacc[8] = {};
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 xu[ROWS], du[ROWS], ru[ROWS], wu = zero;
  if (mine) wu = *reinterpret_cast<const uint4*>(w + c);
  const uint32_t ws[4] = {wu.x, wu.y, wu.z, wu.w};
  float rstd[ROWS];
  auto load = [&](long long first) {               // rows past the end, and columns past the row, are zero
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const long long row = first + static_cast<long long>(k) * gridDim.x;
      xu[k] = du[k] = ru[k] = zero;
      rstd[k] = 0.f;
      if (row >= T) continue;
      rstd[k] = rstd_in[row];
      if (!mine) continue;
      xu[k] = *reinterpret_cast<const uint4*>(x + row * H + c);
      du[k] = *reinterpret_cast<const uint4*>(dy + row * H + c);
      if (dres_in) ru[k] = *reinterpret_cast<const uint4*>(dres_in + row * H + c);
    }
  };
  load(blockIdx.x);
  const long long step = static_cast<long long>(ROWS) * gridDim.x;
  for (long long first = blockIdx.x; first < T; first += WALK ? step : T) {
    float xh[ROWS][8], g[ROWS][8], dot[ROWS], r[ROWS];
    uint4 rs[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const uint32_t xs[4] = {xu[k].x, xu[k].y, xu[k].z, xu[k].w}, ds[4] = {du[k].x, du[k].y, du[k].z, du[k].w};
      const bool there = first + static_cast<long long>(k) * gridDim.x < T;
      rs[k] = ru[k];
      r[k] = rstd[k];
      dot[k] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 xf = unpack_bf16(xs[j]), df = unpack_bf16(ds[j]);
        float2 wf = unpack_bf16(ws[j]);
        if (one_plus_w) { wf.x += 1.f; wf.y += 1.f; }
        const float h0 = xf.x * r[k], h1 = xf.y * r[k];
        xh[k][2 * j] = h0; xh[k][2 * j + 1] = h1;
        g[k][2 * j] = df.x * wf.x; g[k][2 * j + 1] = df.y * wf.y;
        if (mine && (ROWS == 1 || there)) {
          dot[k] += g[k][2 * j] * h0 + g[k][2 * j + 1] * h1;
          dwacc[2 * j] += df.x * h0;
          dwacc[2 * j + 1] += df.y * h1;
        }
      }
    }
    if (WALK) load(first + step);
    block_sums<ROWS>(dot, red);
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const long long row = first + static_cast<long long>(k) * gridDim.x;
      if (!mine || row >= T) continue;
      const float d = dot[k] / static_cast<float>(H);
      const uint32_t res[4] = {rs[k].x, rs[k].y, rs[k].z, rs[k].w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float o0 = r[k] * (g[k][2 * j] - xh[k][2 * j] * d), o1 = r[k] * (g[k][2 * j + 1] - xh[k][2 * j + 1] * d);
        if (dres_in) {
          const float2 a = unpack_bf16(res[j]);
          o0 += a.x; o1 += a.y;
        }
        o[j] = pack_bf16(o0, o1);
      }
      *reinterpret_cast<uint4*>(dx + row * H + c) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  if (mine) {
    float* dst = dw_partial + static_cast<long long>(blockIdx.x) * H + c;
#pragma unroll
    for (int j = 0; j < 8; ++j) dst[j] = dwacc[j];
  }
}

// ============================================================================
// LayerNorm (weight + bias) for the vision tower: fp32 statistics, bf16 in / out.
//   y = (x - mean) * rstd * w + b
//   dx = rstd * (g - mean(g) - xhat * mean(g * xhat)),  g = dy * w ; dw = sum dy * xhat ; db = sum dy
// Forward: one block per row.  Backward: persistent blocks, per-thread dw / db partials flushed to
// part[blockIdx.x][2][H] and reduced by colsum_kernel (deterministic order).
// HF ViT eager `nn.LayerNorm` of the reference's vision blocks (models/qwen3_5/modeling_qwen3_5.py:1035-1207).
// ============================================================================
template <int MAX_ITERS>
__global__ void layernorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                     const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y,
                                     float* __restrict__ mean_out, float* __restrict__ rstd_out, int H, float eps) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  float vals[MAX_ITERS][8];
  float s = 0.f;
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int c = (it * blockDim.x + threadIdx.x) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) vals[it][j] = 0.f;
    if (c >= H) continue;
    const uint4 u = *reinterpret_cast<const uint4*>(x + row * H + c);
    const float2 a = unpack_bf16(u.x), bb = unpack_bf16(u.y), cc = unpack_bf16(u.z), d = unpack_bf16(u.w);
    vals[it][0] = a.x; vals[it][1] = a.y; vals[it][2] = bb.x; vals[it][3] = bb.y;
    vals[it][4] = cc.x; vals[it][5] = cc.y; vals[it][6] = d.x; vals[it][7] = d.y;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += vals[it][j];
  }
  const float mean = block_sum(s, red) / static_cast<float>(H);
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int c = (it * blockDim.x + threadIdx.x) * 8;
    if (c >= H) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float d = vals[it][j] - mean;
      ss += d * d;
    }
  }
  const float rstd = rsqrtf(block_sum(ss, red) / static_cast<float>(H) + eps);
  if (threadIdx.x == 0) {
    mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
#pragma unroll
  for (int it = 0; it < MAX_ITERS; ++it) {
    const int c = (it * blockDim.x + threadIdx.x) * 8;
    if (c >= H) continue;
    const uint4 wu = *reinterpret_cast<const uint4*>(w + c);
    const uint4 bu = *reinterpret_cast<const uint4*>(b + c);
    const uint32_t ws[4] = {wu.x, wu.y, wu.z, wu.w}, bs[4] = {bu.x, bu.y, bu.z, bu.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 wf = unpack_bf16(ws[j]), bf = unpack_bf16(bs[j]);
      o[j] = pack_bf16((vals[it][2 * j] - mean) * rstd * wf.x + bf.x, (vals[it][2 * j + 1] - mean) * rstd * wf.y + bf.y);
    }
    *reinterpret_cast<uint4*>(y + row * H + c) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int ROWS, bool WALK>
__global__ void __launch_bounds__(ROWS == 1 ? 1024 : 256)
layernorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                     const float* __restrict__ mean_in, const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                     float* __restrict__ part, long long T, int H) {
  __shared__ float red[64 * ROWS];
  const int c = threadIdx.x * 8;
  const bool mine = c < H;
  float dwacc[8] = {}, dbacc[8] = {};
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 xu[ROWS], du[ROWS], wu = zero;
  if (mine) wu = *reinterpret_cast<const uint4*>(w + c);
  const uint32_t ws[4] = {wu.x, wu.y, wu.z, wu.w};
  float mean_n[ROWS], rstd_n[ROWS];
  auto load = [&](long long first) {               // rows past the end, and columns past the row, are zero
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const long long row = first + static_cast<long long>(k) * gridDim.x;
      xu[k] = du[k] = zero;
      mean_n[k] = rstd_n[k] = 0.f;
      if (row >= T) continue;
      mean_n[k] = mean_in[row];
      rstd_n[k] = rstd_in[row];
      if (!mine) continue;
      xu[k] = *reinterpret_cast<const uint4*>(x + row * H + c);
      du[k] = *reinterpret_cast<const uint4*>(dy + row * H + c);
    }
  };
  load(blockIdx.x);
  const long long step = static_cast<long long>(ROWS) * gridDim.x;
  for (long long first = blockIdx.x; first < T; first += WALK ? step : T) {
    float xh[ROWS][8], g[ROWS][8], sums[2 * ROWS], rstd[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const uint32_t xs[4] = {xu[k].x, xu[k].y, xu[k].z, xu[k].w}, ds[4] = {du[k].x, du[k].y, du[k].z, du[k].w};
      const bool there = first + static_cast<long long>(k) * gridDim.x < T;
      const float mean = mean_n[k];
      rstd[k] = rstd_n[k];
      float sg = 0.f, sgx = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 xf = unpack_bf16(xs[j]), df = unpack_bf16(ds[j]), wf = unpack_bf16(ws[j]);
        const float h0 = (xf.x - mean) * rstd[k], h1 = (xf.y - mean) * rstd[k];
        xh[k][2 * j] = h0; xh[k][2 * j + 1] = h1;
        g[k][2 * j] = df.x * wf.x; g[k][2 * j + 1] = df.y * wf.y;
        if (mine && (ROWS == 1 || there)) {
          sg += g[k][2 * j] + g[k][2 * j + 1];
          sgx += g[k][2 * j] * h0 + g[k][2 * j + 1] * h1;
          dwacc[2 * j] += df.x * h0; dwacc[2 * j + 1] += df.y * h1;
          dbacc[2 * j] += df.x; dbacc[2 * j + 1] += df.y;
        }
      }
      sums[2 * k] = sg;
      sums[2 * k + 1] = sgx;
    }
    if (WALK) load(first + step);
    block_sums<2 * ROWS>(sums, red);
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const long long row = first + static_cast<long long>(k) * gridDim.x;
      if (!mine || row >= T) continue;
      const float sg = sums[2 * k] / static_cast<float>(H), sgx = sums[2 * k + 1] / static_cast<float>(H);
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        o[j] = pack_bf16(rstd[k] * (g[k][2 * j] - sg - xh[k][2 * j] * sgx), rstd[k] * (g[k][2 * j + 1] - sg - xh[k][2 * j + 1] * sgx));
      *reinterpret_cast<uint4*>(dx + row * H + c) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  if (mine) {
    float* dwp = part + static_cast<long long>(blockIdx.x) * 2 * H + c;
    float* dbp = dwp + H;
#pragma unroll
    for (int j = 0; j < 8; ++j) { dwp[j] = dwacc[j]; dbp[j] = dbacc[j]; }
  }
}

// ============================================================================
// y = act(x + bias) (+ residual): the elementwise tail of a biased projection in one pass.
//   act 0: identity, 1: GELU (tanh approximation), 2: GELU (erf).   x [R, C], bias [C], residual [R, C]; C % 8 == 0
// Backward: dx = dy * act'(x + bias) ; dbias = column sum of dx (partials per block, reduced by colsum_kernel).
// ============================================================================
__device__ __forceinline__ float act_fwd(float v, int act) {
  if (act == 1) {
    const float u = 0.7978845608028654f * (v + 0.044715f * v * v * v);
    return 0.5f * v * (1.f + tanhf(u));
  }
  if (act == 2) return 0.5f * v * (1.f + erff(v * 0.7071067811865476f));
  return v;
}
__device__ __forceinline__ float act_grad(float v, int act) {
  if (act == 1) {
    const float u = 0.7978845608028654f * (v + 0.044715f * v * v * v);
    const float t = tanhf(u);
    return 0.5f * (1.f + t) + 0.5f * v * (1.f - t * t) * 0.7978845608028654f * (1.f + 3.f * 0.044715f * v * v);
  }
  if (act == 2) return 0.5f * (1.f + erff(v * 0.7071067811865476f)) + v * 0.3989422804014327f * __expf(-0.5f * v * v);
  return 1.f;
}

__global__ void bias_act_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ bias,
                                    const __nv_bfloat16* __restrict__ residual, __nv_bfloat16* __restrict__ y,
                                    long long R, int C, int act) {
  const long long vec_per_row = C / 8;
  const long long total = R * vec_per_row;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % vec_per_row) * 8;
    const uint4 xu = *(reinterpret_cast<const uint4*>(x) + i);
    const uint4 bu = *reinterpret_cast<const uint4*>(bias + c);
    uint4 ru = make_uint4(0u, 0u, 0u, 0u);
    if (residual) ru = *(reinterpret_cast<const uint4*>(residual) + i);
    const uint32_t xs[4] = {xu.x, xu.y, xu.z, xu.w}, bs[4] = {bu.x, bu.y, bu.z, bu.w}, rs[4] = {ru.x, ru.y, ru.z, ru.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 xf = unpack_bf16(xs[j]), bf = unpack_bf16(bs[j]), rf = unpack_bf16(rs[j]);
      o[j] = pack_bf16(act_fwd(xf.x + bf.x, act) + rf.x, act_fwd(xf.y + bf.y, act) + rf.y);
    }
    *(reinterpret_cast<uint4*>(y) + i) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// Blocks walk rows of up to 8192 columns (blockIdx.y: which), eight columns a thread, the next row's loads ahead of this one's arithmetic.
// With the column sum, GELU, before -> now: 2850 x 4304 25 -> 21 us, 16384 x 4096 108 -> 74, 2000 x 16384 107 -> 54.  (A form without the
// walk for blocks of one row, as the norms have, takes 4.8 us for 8 x 3456, this one 4.5; 3.6 for 8 x 1152 either way.)
__global__ void __launch_bounds__(1024)
bias_act_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ bias,
                    __nv_bfloat16* __restrict__ dx, float* __restrict__ part, long long R, int C, int act) {
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= C) return;
  float acc[8] = {};
  uint4 du = make_uint4(0, 0, 0, 0), xu = du, bu = du;
  if (act) bu = *reinterpret_cast<const uint4*>(bias + c);
  const uint32_t bs[4] = {bu.x, bu.y, bu.z, bu.w};
  auto load = [&](long long row) {
    if (row >= R) return;
    du = *reinterpret_cast<const uint4*>(dy + row * C + c);
    if (act) xu = *reinterpret_cast<const uint4*>(x + row * C + c);
  };
  load(blockIdx.x);
  for (long long row = blockIdx.x; row < R; row += gridDim.x) {
    const uint32_t ds[4] = {du.x, du.y, du.z, du.w}, xs[4] = {xu.x, xu.y, xu.z, xu.w};
    load(row + gridDim.x);
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 g = unpack_bf16(ds[j]);
      o[j] = ds[j];
      if (act) {
        const float2 xf = unpack_bf16(xs[j]), bf = unpack_bf16(bs[j]);
        g.x *= act_grad(xf.x + bf.x, act);
        g.y *= act_grad(xf.y + bf.y, act);
        o[j] = pack_bf16(g.x, g.y);
      }
      acc[2 * j] += g.x; acc[2 * j + 1] += g.y;
    }
    if (dx) *reinterpret_cast<uint4*>(dx + row * C + c) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  float* dst = part + static_cast<long long>(blockIdx.x) * C + c;
#pragma unroll
  for (int j = 0; j < 8; ++j) dst[j] = acc[j];
}

// ============================================================================
// Causal depthwise short convolution over a packed row (linear-attention mixers: GDN / KDA q, k, v streams).
//   pre[t, c] = bias[c] + sum_{s < W} w[c, W-1-s] * x[t-s, c]   for t-s inside t's sequence;   y = silu(pre) or pre
// x, y: [T, D] bf16 (D % 8 == 0), w: [D, W] bf16 (tap W-1 multiplies the current token), seq_start[t] = first token of
// t's sequence, seq_end[t] = one past its last.  W <= 8.
// Backward: dpre = dy * act'(pre) (pre is recomputed);  dx[t] = sum_s w[., W-1-s] * dpre[t+s] for t+s in the sequence;
// dw[c, W-1-s] = sum_t dpre[t, c] * x[t-s, c];  db = sum_t dpre.  Pass 1 writes dpre (bf16) and per-block dw / db
// partials; pass 2 forms dx (filters of up to four taps do both in one pass).  Torch formulation: ops/providers/native/causal_conv1d.py of the reference (fla Triton
// kernel on its GPU path).
// ============================================================================
constexpr int CONV_MAX_W = 8;   // widest supported filter

// Filters of up to four taps (every linear-attention layer): a thread owns 4 channels (8 would spill the window), walks its rows four
// at a time with the next four rows' loads already issued, and keeps the taps' window in registers, so that x (and dy) are read
// once.  One pass each way: the backward adds every dpre row into the W rows of dx that it reaches while they are still in registers
// (the W - 1 rows behind a block are recomputed by it), which saves writing and re-reading dpre.  Steps in which every tap of every row
// counts run without the checks, and products go two channels at a time.  The next rows' loads have to be held in place: as plain
// conditional loads they drew the unpacking of their row with them, so that a thread waited for memory at every step, which was most of
// the backward's time.  What bounds it now is the issue of its arithmetic (two exponentials and 48 products per element pair).
// 4096 x 8192, W = 4, from cold caches with the column sums: forward 47 -> 41 us, backward 132 -> 79; 16384 x 6144: 121 -> 100 and
// 343 -> 179; 2047 x 3072: 16 and 50 -> 36 (memory alone: 22 and 33 us for the first).
constexpr int CONV_ROWS = 4;    // rows per step

__device__ __forceinline__ void unpack4(const uint2& u, float (&f)[4]) {
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&f)[4]) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
}

// Loads that stay where they are written: the compiler otherwise moves the unpacking of a row up to its load, and the thread waits there
__device__ __forceinline__ uint2 load_here(const __nv_bfloat16* p) {
  uint2 v;
  asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ int load_here(const int* p) {
  int v;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// c += a * b for two neighbouring channels (one instruction; each half rounds as an fma of its own)
__device__ __forceinline__ void fma2(float& c0, float& c1, float a0, float a1, float b0, float b1) {
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%0, %1};\n\t"
      "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "+f"(c0), "+f"(c1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ void fma4(float (&c)[4], const float (&a)[4], const float (&b)[4]) {
  fma2(c[0], c[1], a[0], a[1], b[0], b[1]);
  fma2(c[2], c[3], a[2], a[3], b[2], b[3]);
}

template <bool BWD>
__global__ void __launch_bounds__(128, BWD ? 4 : 6)
causal_conv1d_w4_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                        const __nv_bfloat16* __restrict__ bias, const int* __restrict__ seq_start,
                        const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ out,
                        float* __restrict__ part, long long T, int D, int W, int silu, int rows_per_block) {
  constexpr int WM = 4;
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (c >= D) return;
  float wt[WM][4];   // wt[s] = tap for distance s into the past
#pragma unroll
  for (int s = 0; s < WM; ++s)
#pragma unroll
    for (int j = 0; j < 4; ++j) wt[s][j] = (s < W) ? __bfloat162float(w[static_cast<long long>(c + j) * W + (W - 1 - s)]) : 0.f;
  float bs[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) bs[j] = bias ? __bfloat162float(bias[c + j]) : 0.f;
  float dwacc[BWD ? WM : 1][4], dbacc[BWD ? 4 : 1], acc[BWD ? WM : 1][4];   // acc[s]: dx of the row s behind the current one
  if (BWD) {
#pragma unroll
    for (int s = 0; s < WM; ++s)
#pragma unroll
      for (int j = 0; j < 4; ++j) dwacc[s][j] = acc[s][j] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) dbacc[j] = 0.f;
  }
  const long long r0 = static_cast<long long>(blockIdx.y) * rows_per_block;
  const long long r1 = (r0 + rows_per_block < T) ? r0 + rows_per_block : T;
  const long long re = BWD ? ((r1 + W - 1 < T) ? r1 + W - 1 : T) : r1;      // rows computed, the halo included
  const uint2 zero = make_uint2(0, 0);
  uint2 hist[WM - 1];   // x of the rows 1 .. W - 1 behind
#pragma unroll
  for (int s = 1; s < WM; ++s)
    hist[s - 1] = (s < W && r0 >= s) ? *reinterpret_cast<const uint2*>(x + (r0 - s) * D + c) : zero;
  uint2 nx[CONV_ROWS], ng[CONV_ROWS];
  int nf[CONV_ROWS];
  auto fetch = [&](long long t0) {
#pragma unroll
    for (int u = 0; u < CONV_ROWS; ++u) {
      const long long t = t0 + u < re ? t0 + u : re - 1;     // (rows from `re` on are loaded for nothing)
      nx[u] = load_here(x + t * D + c);
      if (BWD) ng[u] = load_here(dy + t * D + c);
      nf[u] = load_here(seq_start + t);
    }
  };
  fetch(r0);
  for (long long t0 = r0; t0 < re; t0 += CONV_ROWS) {
    uint2 cx[CONV_ROWS], cg[CONV_ROWS];
    int cf[CONV_ROWS];
#pragma unroll
    for (int u = 0; u < CONV_ROWS; ++u) {
      cx[u] = nx[u];
      if (BWD) cg[u] = ng[u];
      cf[u] = nf[u];
    }
    if (t0 + CONV_ROWS < re) fetch(t0 + CONV_ROWS);
    // INNER: all four taps of all four rows lie in their sequences, the rows are this block's and so are the rows they complete
    auto row = [&](auto inner, int u) {
      constexpr bool INNER = decltype(inner)::value;
      const long long t = t0 + u;
      if (!INNER && t >= re) return;
      const int reach = static_cast<int>(t - cf[u] < WM ? t - cf[u] : WM);   // how far back the sequence goes, at most WM
      float xs[WM][4], pre[4];
      unpack4(cx[u], xs[0]);
#pragma unroll
      for (int j = 0; j < 4; ++j) pre[j] = bs[j];
      fma4(pre, wt[0], xs[0]);
#pragma unroll
      for (int s = 1; s < WM; ++s) {
        unpack4(hist[s - 1], xs[s]);
        if (INNER || (s <= reach && s < W)) {      // (not a product with zero: rows and taps may be infinite)
          fma4(pre, wt[s], xs[s]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) xs[s][j] = 0.f;
        }
      }
      if (!BWD) {
        float o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = silu ? pre[j] / (1.f + __expf(-pre[j])) : pre[j];
        store4(out + t * D + c, o);
      } else {
        float d[4];
        unpack4(cg[u], d);
        if (silu) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float sg = 1.f / (1.f + __expf(-pre[j]));
            d[j] *= sg * (1.f + pre[j] * (1.f - sg));
          }
        }
        if (INNER || t < r1) {
#pragma unroll
          for (int j = 0; j < 4; ++j) dbacc[j] += d[j];
#pragma unroll
          for (int s = 0; s < WM; ++s) fma4(dwacc[s], d, xs[s]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          d[j] = __bfloat162float(__float2bfloat16(d[j]));
          acc[0][j] = wt[0][j] * d[j];
        }
        // this row reaches the dx of the rows up to W - 1 behind it in its sequence
#pragma unroll
        for (int s = 1; s < WM; ++s)
          if (INNER || (s <= reach && s < W)) fma4(acc[s], wt[s], d);
        const long long done = t - (WM - 1);        // no later row reaches it
        if (INNER || (done >= r0 && done < r1)) store4(out + done * D + c, acc[WM - 1]);
#pragma unroll
        for (int s = WM - 1; s > 0; --s)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[s][j] = acc[s - 1][j];
      }
#pragma unroll
      for (int s = WM - 2; s > 0; --s) hist[s] = hist[s - 1];
      hist[0] = cx[u];
    };
    bool inner = W == WM && t0 + CONV_ROWS <= r1 && (!BWD || t0 >= r0 + WM - 1);
#pragma unroll
    for (int u = 0; u < CONV_ROWS; ++u) inner = inner && t0 + u - cf[u] >= WM - 1;
    if (inner) {
#pragma unroll
      for (int u = 0; u < CONV_ROWS; ++u) row(std::true_type{}, u);
    } else {
#pragma unroll
      for (int u = 0; u < CONV_ROWS; ++u) row(std::false_type{}, u);
    }
  }
  if (BWD) {
    // the rows behind the last computed one (acc has moved on by one: acc[s] is the dx of row re - s)
#pragma unroll
    for (int s = WM - 1; s > 0; --s) {
      const long long row = re - s;
      if (row >= r0 && row < r1) store4(out + row * D + c, acc[s]);
    }
    // part[blockIdx.y][(W + 1)][D]: W tap planes (distance s) then the bias plane
    float* base = part + static_cast<long long>(blockIdx.y) * (W + 1) * D;
#pragma unroll
    for (int s = 0; s < WM; ++s)
      if (s < W)
#pragma unroll
        for (int j = 0; j < 4; ++j) base[static_cast<long long>(s) * D + c + j] = dwacc[s][j];
#pragma unroll
    for (int j = 0; j < 4; ++j) base[static_cast<long long>(W) * D + c + j] = dbacc[j];
  }
}

// grid: (ceil(D/8 / blockDim.x), row blocks); each thread owns 8 channels and walks rows [r0, r1)
template <bool BWD, int WMAX>
__global__ void causal_conv1d_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                     const __nv_bfloat16* __restrict__ bias, const int* __restrict__ seq_start,
                                     const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ out,
                                     float* __restrict__ part, long long T, int D, int W, int silu, int rows_per_block) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= D) return;
  float wt[WMAX][8];   // wt[s] = tap for distance s into the past
#pragma unroll
  for (int s = 0; s < WMAX; ++s)
#pragma unroll
    for (int j = 0; j < 8; ++j) wt[s][j] = (s < W) ? __bfloat162float(w[static_cast<long long>(c + j) * W + (W - 1 - s)]) : 0.f;
  float bs[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) bs[j] = bias ? __bfloat162float(bias[c + j]) : 0.f;
  float dwacc[WMAX][8], dbacc[8];
  if (BWD) {
#pragma unroll
    for (int s = 0; s < WMAX; ++s)
#pragma unroll
      for (int j = 0; j < 8; ++j) dwacc[s][j] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) dbacc[j] = 0.f;
  }
  const long long r0 = static_cast<long long>(blockIdx.y) * rows_per_block;
  const long long r1 = (r0 + rows_per_block < T) ? r0 + rows_per_block : T;
  for (long long t = r0; t < r1; ++t) {
    const long long first = seq_start[t];
    float xs[WMAX][8];
    float pre[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) pre[j] = bs[j];
#pragma unroll
    for (int s = 0; s < WMAX; ++s) {
      if (s < W && t - s >= first) {
        load8(x + (t - s) * D + c, xs[s]);
#pragma unroll
        for (int j = 0; j < 8; ++j) pre[j] += wt[s][j] * xs[s][j];
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) xs[s][j] = 0.f;
      }
    }
    float o[8];
    if (!BWD) {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = silu ? pre[j] / (1.f + __expf(-pre[j])) : pre[j];
    } else {
      float g[8];
      load8(dy + t * D + c, g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float d = g[j];
        if (silu) {
          const float sg = 1.f / (1.f + __expf(-pre[j]));
          d *= sg * (1.f + pre[j] * (1.f - sg));
        }
        o[j] = d;
        dbacc[j] += d;
#pragma unroll
        for (int s = 0; s < WMAX; ++s) dwacc[s][j] += d * xs[s][j];
      }
    }
    store8(out + t * D + c, o);
  }
  if (BWD) {
    // part[blockIdx.y][(W + 1)][D]: W tap planes (distance s) then the bias plane
    float* base = part + static_cast<long long>(blockIdx.y) * (W + 1) * D;
#pragma unroll
    for (int s = 0; s < WMAX; ++s)
      if (s < W)
#pragma unroll
        for (int j = 0; j < 8; ++j) base[static_cast<long long>(s) * D + c + j] = dwacc[s][j];
#pragma unroll
    for (int j = 0; j < 8; ++j) base[static_cast<long long>(W) * D + c + j] = dbacc[j];
  }
}

// dx[t] = sum_s w[., W-1-s] * dpre[t+s] for t+s < seq_end[t]
template <int WMAX>
__global__ void causal_conv1d_dx_kernel(const __nv_bfloat16* __restrict__ dpre, const __nv_bfloat16* __restrict__ w,
                                        const int* __restrict__ seq_end, __nv_bfloat16* __restrict__ dx, long long T,
                                        int D, int W, int rows_per_block) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= D) return;
  float wt[WMAX][8];
#pragma unroll
  for (int s = 0; s < WMAX; ++s)
#pragma unroll
    for (int j = 0; j < 8; ++j) wt[s][j] = (s < W) ? __bfloat162float(w[static_cast<long long>(c + j) * W + (W - 1 - s)]) : 0.f;
  const long long r0 = static_cast<long long>(blockIdx.y) * rows_per_block;
  const long long r1 = (r0 + rows_per_block < T) ? r0 + rows_per_block : T;
  for (long long t = r0; t < r1; ++t) {
    const long long last = seq_end[t];
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int s = 0; s < WMAX; ++s) {
      if (s < W && t + s < last) {
        float g[8];
        load8(dpre + (t + s) * D + c, g);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += wt[s][j] * g[j];
      }
    }
    store8(dx + t * D + c, acc);
  }
}

// ============================================================================
// Fused per-head RMSNorm + rotary embedding (half rotation) for q and k.
// in : qkv [T, ld] bf16 with q heads at column 0, k heads at column Hq*D
// out: q_out [T, Hq, D], k_out [T, Hk, D]  (v is consumed in place by attention)
// cos/sin: [T, D/2] fp32.  D == 128.
// Forward: sixteen lanes per (token, head), a lane owns channels 4l .. 4l + 3 of both halves, so that every load moves 8 bytes
// (a whole warp per head moved 4: 30 us for 4096 tokens x 36 heads, 21 now, 80 MB).  Backward: a whole warp per (token, head);
// the same split there doubles the weight-gradient accumulators per thread and took 48 us instead of 41.
// ============================================================================
__device__ __forceinline__ void qk_load4(const __nv_bfloat16* p, float (&f)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
__device__ __forceinline__ void qk_store4(__nv_bfloat16* p, const float (&f)[4]) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
}
__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float bf16_rounded(float v) { return __bfloat162float(__float2bfloat16(v)); }

__global__ void __launch_bounds__(256)
qknorm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, long long ld, int Hq, int Hk,
                       const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk,
                       const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                       __nv_bfloat16* __restrict__ q_out, __nv_bfloat16* __restrict__ k_out,
                       float* __restrict__ rstd_out, long long T, float eps, int use_norm) {
  constexpr int D = 128;
  const int l = threadIdx.x & 15;
  const int heads = Hq + Hk;
  const long long total = T * heads;
  long long item = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 4;
  // the two halves of a warp shuffle together: the last odd item is computed twice and stored once
  const bool ok = item < total;
  if (!ok) item = total - 1;
  const long long t = item / heads;
  const int h = static_cast<int>(item - t * heads);
  const bool is_q = h < Hq;
  const __nv_bfloat16* src = qkv + t * ld + static_cast<long long>(h) * D;
  const __nv_bfloat16* w = is_q ? wq : wk;
  __nv_bfloat16* dst = is_q ? q_out + (t * Hq + h) * D : k_out + (t * Hk + (h - Hq)) * D;
  float lo[4], hi[4];
  qk_load4(src + 4 * l, lo);
  qk_load4(src + 64 + 4 * l, hi);
  const float4 c4 = __ldg(reinterpret_cast<const float4*>(cos_t + t * (D / 2)) + l);
  const float4 s4 = __ldg(reinterpret_cast<const float4*>(sin_t + t * (D / 2)) + l);
  const float c[4] = {c4.x, c4.y, c4.z, c4.w}, s[4] = {s4.x, s4.y, s4.z, s4.w};
  float rstd = 1.f;
  if (use_norm) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) ss += lo[j] * lo[j] + hi[j] * hi[j];
    rstd = rsqrtf(half_warp_sum(ss) / D + eps);
    float wl[4], wh[4];
    qk_load4(w + 4 * l, wl);
    qk_load4(w + 64 + 4 * l, wh);
#pragma unroll
    for (int j = 0; j < 4; ++j) {   // the normalised tensor is a bf16 tensor in the eager formulation
      lo[j] = bf16_rounded(bf16_rounded(lo[j] * rstd) * wl[j]);
      hi[j] = bf16_rounded(bf16_rounded(hi[j] * rstd) * wh[j]);
    }
  }
  if (!ok) return;
  if (rstd_out && l == 0) rstd_out[item] = rstd;
  float o_lo[4], o_hi[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    o_lo[j] = lo[j] * c[j] - hi[j] * s[j];
    o_hi[j] = hi[j] * c[j] + lo[j] * s[j];
  }
  qk_store4(dst + 4 * l, o_lo);
  qk_store4(dst + 64 + 4 * l, o_hi);
}

// Backward: given dq_out / dk_out, the pre-norm qkv and rstd -> the q and k columns of d(qkv), with `dv` the v columns too, and
// the weight gradients' partial sums, part[block][2][128] (added up by colsum in a fixed order).  A warp takes four heads of a
// token at a time: one fetch of the angles, and the loads of four heads in flight instead of one (bound by latency before:
// 4096 tokens x 36 heads 41 us, now 34 and 4 for the sums).  The value columns ride along for the launch and the pass that a copy costs.
constexpr int QKB_HEADS = 4;
__global__ void __launch_bounds__(256)
qknorm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk, const __nv_bfloat16* __restrict__ dv,
                       const __nv_bfloat16* __restrict__ qkv, long long ld, int Hq, int Hk, const __nv_bfloat16* __restrict__ wq,
                       const __nv_bfloat16* __restrict__ wk, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                       const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dqkv, long long ldd, float* __restrict__ part,
                       long long T, int use_norm) {
  constexpr int D = 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int heads = Hq + Hk, all = dv ? heads + Hk : heads, groups = (all + QKB_HEADS - 1) / QKB_HEADS;
  const long long nwarps = static_cast<long long>(gridDim.x) * 8;
  float accq[4] = {0, 0, 0, 0}, acck[4] = {0, 0, 0, 0};
  for (long long unit = static_cast<long long>(blockIdx.x) * 8 + warp; unit < T * groups; unit += nwarps) {
    const long long t = unit / groups;
    const int h0 = static_cast<int>(unit - t * groups) * QKB_HEADS;
    uint32_t glo[QKB_HEADS], ghi[QKB_HEADS], xlo[QKB_HEADS], xhi[QKB_HEADS];
    float rs[QKB_HEADS];
#pragma unroll
    for (int u = 0; u < QKB_HEADS; ++u) {
      const int h = h0 + u;
      glo[u] = ghi[u] = xlo[u] = xhi[u] = 0u;
      rs[u] = 1.f;
      if (h >= all) continue;
      const __nv_bfloat16* g = h < Hq ? dq + (t * Hq + h) * D : h < heads ? dk + (t * Hk + (h - Hq)) * D : dv + (t * Hk + (h - heads)) * D;
      glo[u] = *reinterpret_cast<const uint32_t*>(g + 2 * lane);
      ghi[u] = *reinterpret_cast<const uint32_t*>(g + 64 + 2 * lane);
      if (use_norm && h < heads) {
        const __nv_bfloat16* src = qkv + t * ld + static_cast<long long>(h) * D;
        xlo[u] = *reinterpret_cast<const uint32_t*>(src + 2 * lane);
        xhi[u] = *reinterpret_cast<const uint32_t*>(src + 64 + 2 * lane);
        rs[u] = rstd_in[t * heads + h];
      }
    }
    const float2 c = *reinterpret_cast<const float2*>(cos_t + t * (D / 2) + 2 * lane);
    const float2 s = *reinterpret_cast<const float2*>(sin_t + t * (D / 2) + 2 * lane);
#pragma unroll
    for (int u = 0; u < QKB_HEADS; ++u) {
      const int h = h0 + u;
      if (h >= all) continue;
      __nv_bfloat16* out = dqkv + t * ldd + static_cast<long long>(h) * D;
      if (h < heads) {
        const float2 gl = unpack_bf16(glo[u]), gh = unpack_bf16(ghi[u]);
        // inverse rotation (transpose of the forward map)
        float dl_x = gl.x * c.x + gh.x * s.x, dl_y = gl.y * c.y + gh.y * s.y;
        float dh_x = gh.x * c.x - gl.x * s.x, dh_y = gh.y * c.y - gl.y * s.y;
        if (use_norm) {
          const bool is_q = h < Hq;
          const __nv_bfloat16* w = is_q ? wq : wk;
          const float2 xl = unpack_bf16(xlo[u]), xr = unpack_bf16(xhi[u]);
          const float2 wl = unpack_bf16(*reinterpret_cast<const uint32_t*>(w + 2 * lane));
          const float2 wh = unpack_bf16(*reinterpret_cast<const uint32_t*>(w + 64 + 2 * lane));
          const float rstd = rs[u];
          const float xh[4] = {xl.x * rstd, xl.y * rstd, xr.x * rstd, xr.y * rstd};
          const float dyv[4] = {dl_x, dl_y, dh_x, dh_y};
          const float wv[4] = {wl.x, wl.y, wh.x, wh.y};
          float gg[4];
          float dot = 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            gg[j] = dyv[j] * wv[j];
            dot += gg[j] * xh[j];
            if (is_q) accq[j] += dyv[j] * xh[j]; else acck[j] += dyv[j] * xh[j];
          }
          dot = warp_sum(dot) / D;
          dl_x = rstd * (gg[0] - xh[0] * dot); dl_y = rstd * (gg[1] - xh[1] * dot);
          dh_x = rstd * (gg[2] - xh[2] * dot); dh_y = rstd * (gg[3] - xh[3] * dot);
        }
        glo[u] = pack_bf16(dl_x, dl_y);
        ghi[u] = pack_bf16(dh_x, dh_y);
      }
      *reinterpret_cast<uint32_t*>(out + 2 * lane) = glo[u];
      *reinterpret_cast<uint32_t*>(out + 64 + 2 * lane) = ghi[u];
    }
  }
  if (use_norm) {
    __shared__ float sdw[8][2][D];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = (j >> 1) * 64 + 2 * lane + (j & 1);
      sdw[warp][0][col] = accq[j];
      sdw[warp][1][col] = acck[j];
    }
    __syncthreads();
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += (&sdw[w][0][0])[threadIdx.x];
    part[static_cast<long long>(blockIdx.x) * 2 * D + threadIdx.x] = v;
  }
}

// ============================================================================
// Half-rotation RoPE of [T, heads, 2 * half] with any token / head stride; y contiguous.  sign = -1 is the transpose (the
// backward).  Four pairs per thread, fp32 arithmetic, one rounding.  3000 patches x 16 heads of 72: 5.5 us each, in place of about
// ten torch launches forward and more backward.
//   y1 = x1 c - sign x2 s,  y2 = x2 c + sign x1 s
// ============================================================================
__global__ void rope_kernel(const __nv_bfloat16* __restrict__ x, long long x_t, long long x_h, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, __nv_bfloat16* __restrict__ y, long long total, int heads, int half,
                            float sign) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int q = half / 4;
  const long long th = idx / q;
  const int c = static_cast<int>(idx - th * q) * 4;
  const long long t = th / heads;
  const int h = static_cast<int>(th - t * heads);
  const __nv_bfloat16* src = x + t * x_t + h * x_h + c;
  const uint2 u1 = *reinterpret_cast<const uint2*>(src), u2 = *reinterpret_cast<const uint2*>(src + half);
  const float4 co = __ldg(reinterpret_cast<const float4*>(cos_t + t * half + c));
  float4 si = __ldg(reinterpret_cast<const float4*>(sin_t + t * half + c));
  si.x *= sign; si.y *= sign; si.z *= sign; si.w *= sign;
  const float2 a0 = unpack_bf16(u1.x), a1 = unpack_bf16(u1.y), b0 = unpack_bf16(u2.x), b1 = unpack_bf16(u2.y);
  __nv_bfloat16* dst = y + th * 2 * half + c;
  *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(a0.x * co.x - b0.x * si.x, a0.y * co.y - b0.y * si.y),
                                              pack_bf16(a1.x * co.z - b1.x * si.z, a1.y * co.w - b1.y * si.w));
  *reinterpret_cast<uint2*>(dst + half) = make_uint2(pack_bf16(b0.x * co.x + a0.x * si.x, b0.y * co.y + a0.y * si.y),
                                                     pack_bf16(b1.x * co.z + a1.x * si.z, b1.y * co.w + a1.y * si.w));
}

// ============================================================================
// Between a biased QKV projection and full attention (vision blocks): x [T, 3, heads, 2 half], bias of a row's width ->
// q, k = RoPE(x + bias) and v = x + bias, each [T, heads, 2 half], with x + bias rounded to bf16 first (the value that a separate
// pass stores).  Backward: dx [T, 3, heads, 2 half] from the three gradients, and the bias gradient as partial column sums of the
// rounded dx.  A thread keeps ITEMS fixed groups of four pairs (columns c .. c + 3 and half + c ..) over all rows of its block, so
// that bias and sums stay in registers.  2850 patches and 16 heads of 72 (40 MB each way): 15 and 19 us, where passes of their own
// (bias, two rotations, a copy of v; backward two rotations, three cleared buffers, three copies into them, two sums, bias) took
// 30 and 117 in 16 launches.
// ============================================================================
template <int ITEMS, bool BACK>
__global__ void qkv_rope_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ bias, const float* __restrict__ cos_t,
                                const float* __restrict__ sin_t, __nv_bfloat16* q, __nv_bfloat16* k, __nv_bfloat16* v,
                                __nv_bfloat16* __restrict__ dx, float* __restrict__ part, long long T, int heads, int half) {
  const int per = half / 4, row = heads * 2 * half;      // groups of a head; elements of q's (k's, v's) row
  int col[ITEMS], which[ITEMS], ang[ITEMS];              // first column of the group in its third, the third, its first angle
  uint2 b1[ITEMS], b2[ITEMS];
  float acc[ITEMS][8];
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    const int i = it * blockDim.x + threadIdx.x, third = heads * per;
    which[it] = i / third;                               // 3 and more: no group
    const int g = i - which[it] * third, h = g / per;
    ang[it] = (g - h * per) * 4;
    col[it] = h * 2 * half + ang[it];
    b1[it] = b2[it] = make_uint2(0u, 0u);
    if (!BACK && which[it] < 3) {
      b1[it] = *reinterpret_cast<const uint2*>(bias + which[it] * row + col[it]);
      b2[it] = *reinterpret_cast<const uint2*>(bias + which[it] * row + col[it] + half);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[it][j] = 0.f;
  }
  for (long long t = blockIdx.x; t < T; t += gridDim.x) {
    uint2 u1[ITEMS], u2[ITEMS];
    float4 co[ITEMS], si[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      if (which[it] >= 3) continue;
      __nv_bfloat16* part_of = which[it] == 0 ? q : which[it] == 1 ? k : v;
      const __nv_bfloat16* src = BACK ? part_of + t * row + col[it] : x + (3 * t + which[it]) * row + col[it];
      u1[it] = *reinterpret_cast<const uint2*>(src);
      u2[it] = *reinterpret_cast<const uint2*>(src + half);
      if (which[it] < 2) {
        co[it] = __ldg(reinterpret_cast<const float4*>(cos_t + t * half + ang[it]));
        si[it] = __ldg(reinterpret_cast<const float4*>(sin_t + t * half + ang[it]));
      }
    }
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      if (which[it] >= 3) continue;
      uint2 o1 = u1[it], o2 = u2[it];
      if (!BACK) {
        auto add = [](uint32_t a, uint32_t b) {
          const float2 x2 = unpack_bf16(a), y2 = unpack_bf16(b);
          return pack_bf16(x2.x + y2.x, x2.y + y2.y);
        };
        o1 = make_uint2(add(o1.x, b1[it].x), add(o1.y, b1[it].y));
        o2 = make_uint2(add(o2.x, b2[it].x), add(o2.y, b2[it].y));
      }
      if (which[it] < 2) {
        const float4 c = co[it];
        float4 s = si[it];
        if (BACK) { s.x = -s.x; s.y = -s.y; s.z = -s.z; s.w = -s.w; }
        const float2 a0 = unpack_bf16(o1.x), a1 = unpack_bf16(o1.y), e0 = unpack_bf16(o2.x), e1 = unpack_bf16(o2.y);
        o1 = make_uint2(pack_bf16(a0.x * c.x - e0.x * s.x, a0.y * c.y - e0.y * s.y), pack_bf16(a1.x * c.z - e1.x * s.z, a1.y * c.w - e1.y * s.w));
        o2 = make_uint2(pack_bf16(e0.x * c.x + a0.x * s.x, e0.y * c.y + a0.y * s.y), pack_bf16(e1.x * c.z + a1.x * s.z, e1.y * c.w + a1.y * s.w));
      }
      if (BACK) {
        const uint32_t w[4] = {o1.x, o1.y, o2.x, o2.y};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16(w[j]);
          acc[it][2 * j] += f.x;
          acc[it][2 * j + 1] += f.y;
        }
      }
      __nv_bfloat16* part_of = which[it] == 0 ? q : which[it] == 1 ? k : v;
      __nv_bfloat16* dst = BACK ? dx + (3 * t + which[it]) * row + col[it] : part_of + t * row + col[it];
      *reinterpret_cast<uint2*>(dst) = o1;
      *reinterpret_cast<uint2*>(dst + half) = o2;
    }
  }
  if (BACK) {
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      if (which[it] >= 3) continue;
      float* dst = part + static_cast<long long>(blockIdx.x) * 3 * row + which[it] * row + col[it];
      *reinterpret_cast<float4*>(dst) = make_float4(acc[it][0], acc[it][1], acc[it][2], acc[it][3]);
      *reinterpret_cast<float4*>(dst + half) = make_float4(acc[it][4], acc[it][5], acc[it][6], acc[it][7]);
    }
  }
}

// ============================================================================
// SwiGLU (standalone).  x: [R, 2F] = [gate | up]; y: [R, F]; optional row_scale [R].
// ============================================================================
// `nrows` (optional, device): rows at or beyond *nrows are skipped (padded buffers whose fill is only known on the device)
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, __nv_bfloat16* __restrict__ y,
                                  long long ldy, const float* __restrict__ row_scale, long long R, int F,
                                  const int* __restrict__ nrows) {
  const long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
  const long long total = R * F;
  if (idx >= total) return;
  const long long r = idx / F;
  if (nrows && r >= *nrows) return;
  const int c = static_cast<int>(idx - r * F);
  const float sc = row_scale ? row_scale[r] : 1.f;
  uint4 g = *reinterpret_cast<const uint4*>(x + r * ldx + c);
  uint4 u = *reinterpret_cast<const uint4*>(x + r * ldx + F + c);
  uint32_t gs[4] = {g.x, g.y, g.z, g.w}, us[4] = {u.x, u.y, u.z, u.w}, os[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 gf = unpack_bf16(gs[j]), uf = unpack_bf16(us[j]);
    os[j] = pack_bf16(gf.x / (1.f + __expf(-gf.x)) * uf.x * sc, gf.y / (1.f + __expf(-gf.y)) * uf.y * sc);
  }
  *reinterpret_cast<uint4*>(y + r * ldy + c) = make_uint4(os[0], os[1], os[2], os[3]);
}

// Backward: one block per row (so the per-row d(scale) reduction is local).
//   a = silu(g) * u ; y = a * s
//   dg = dy * s * u * sig(g) * (1 + g * (1 - sig(g))) ; du = dy * s * silu(g) ; ds = sum(dy * a)
// `y_out` (optional) receives the forward result again: a caller that needs it for a weight gradient saves the second read
// of x (49152 rows of 768: 37 us for that pass,
// 6 us for the extra output).
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dy, long long lddy,
                                  const __nv_bfloat16* __restrict__ x, long long ldx,
                                  const float* __restrict__ row_scale, __nv_bfloat16* __restrict__ dx, long long lddx,
                                  float* __restrict__ dscale, __nv_bfloat16* __restrict__ y_out, long long ldy, int F,
                                  const int* __restrict__ nrows) {
  __shared__ float red[32];
  const long long r = blockIdx.x;
  if (nrows && r >= *nrows) return;
  const float sc = row_scale ? row_scale[r] : 1.f;
  float ds = 0.f;
  for (int c = threadIdx.x * 8; c < F; c += blockDim.x * 8) {
    uint4 g = *reinterpret_cast<const uint4*>(x + r * ldx + c);
    uint4 u = *reinterpret_cast<const uint4*>(x + r * ldx + F + c);
    uint4 d = *reinterpret_cast<const uint4*>(dy + r * lddy + c);
    uint32_t gs[4] = {g.x, g.y, g.z, g.w}, us[4] = {u.x, u.y, u.z, u.w}, dsrc[4] = {d.x, d.y, d.z, d.w};
    uint32_t og[4], ou[4], oy[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 gf = unpack_bf16(gs[j]), uf = unpack_bf16(us[j]), df = unpack_bf16(dsrc[j]);
      const float den0 = 1.f + __expf(-gf.x), den1 = 1.f + __expf(-gf.y);
      float sg0 = 1.f / den0, sg1 = 1.f / den1;
      oy[j] = pack_bf16(gf.x / den0 * uf.x * sc, gf.y / den1 * uf.y * sc);
      float si0 = gf.x * sg0, si1 = gf.y * sg1;
      ds += df.x * si0 * uf.x + df.y * si1 * uf.y;
      float d0 = df.x * sc, d1 = df.y * sc;
      og[j] = pack_bf16(d0 * uf.x * sg0 * (1.f + gf.x * (1.f - sg0)), d1 * uf.y * sg1 * (1.f + gf.y * (1.f - sg1)));
      ou[j] = pack_bf16(d0 * si0, d1 * si1);
    }
    *reinterpret_cast<uint4*>(dx + r * lddx + c) = make_uint4(og[0], og[1], og[2], og[3]);
    *reinterpret_cast<uint4*>(dx + r * lddx + F + c) = make_uint4(ou[0], ou[1], ou[2], ou[3]);
    if (y_out) *reinterpret_cast<uint4*>(y_out + r * ldy + c) = make_uint4(oy[0], oy[1], oy[2], oy[3]);
  }
  if (dscale) {
    ds = block_sum(ds, red);
    if (threadIdx.x == 0) dscale[r] = ds;
  }
}

// ============================================================================
// Cross-entropy over logits [R, V] (bf16 or fp32), labels int64, ignore_index < 0.
// Writes per-row loss (0 for ignored rows) and, when dlogits != nullptr, the gradient
// (softmax - onehot) * grad_scale[0] in bf16 (may alias a bf16 logits buffer).
// Bound by memory: the rows in flight (two blocks per SM, 90 MB of 151936 logits) and the gradients just written share the L2, and what a
// row's second pass finds there no more is read again.  Where that happens (LONG) the pass walks the row from its end, where it was read
// last, and marks what it reads and writes as the first to leave: 4096 x 151936 bf16, gradient in place, 518 -> 473 us (from the end
// alone 489, marks alone 488; one read and one write at the rate of a copy: 408), 1024 rows 148 -> 133.  Shorter rows are still there,
// and the plain order is the faster one: in place, plain and LONG, 4096 x 32000 111 and 113 us, x 80000 245 and 257, x 112000 350 and
// 356, x 116000 373 and 371, x 128256 411 and 403; with a gradient of its own, which takes L2 as well, x 80000 249 and 256, x 84000 270
// and 268, x 100352 328 and 311 (300 to 600 rows whose logits and gradients just fill the L2 are an exception: 600 x 40000 27.0 and
// 25.7).  With a third fewer instructions it takes the same time; 512 threads per block take 514 us, and 102 with
// 32000 logits.
// ============================================================================
template <typename TL>
__device__ __forceinline__ float ld_logit(const TL* p, long long i);
template <>
__device__ __forceinline__ float ld_logit<float>(const float* p, long long i) { return p[i]; }
template <>
__device__ __forceinline__ float ld_logit<__nv_bfloat16>(const __nv_bfloat16* p, long long i) {
  return __bfloat162float(p[i]);
}

constexpr int CE_THREADS = 1024;
static bool ce_long(int V, bool in_place) { return V >= (in_place ? 114000 : 84000); }      // the measured lines, above
template <typename TL, bool LONG>
__global__ void __launch_bounds__(CE_THREADS)
cross_entropy_kernel(const TL* __restrict__ logits, long long ldl, const long long* __restrict__ labels,
                     float* __restrict__ loss_rows, float* __restrict__ lse_rows, __nv_bfloat16* dlogits, long long ldd,
                     const float* __restrict__ grad_scale, float grad_scale_host, int V) {
  __shared__ float red[32];
  const long long r = blockIdx.x;
  const TL* lr = logits + r * ldl;
  const long long label = labels[r];
  const bool valid = label >= 0 && label < V;
  constexpr bool kBf16 = sizeof(TL) == 2;
  // 16-byte vector path for bf16 rows (8 logits per access); everything else goes element by element
  const bool vec = kBf16 && (V % 8 == 0) && ((reinterpret_cast<uintptr_t>(lr) & 15) == 0) &&
                   (dlogits == nullptr || (reinterpret_cast<uintptr_t>(dlogits + r * ldd) & 15) == 0);
  if (!valid) {
    if (threadIdx.x == 0) { loss_rows[r] = 0.f; if (lse_rows) lse_rows[r] = 0.f; }
    if (dlogits) {
      if (vec) {
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (int c = threadIdx.x * 8; c < V; c += CE_THREADS * 8) *reinterpret_cast<uint4*>(dlogits + r * ldd + c) = z;
      } else {
        __nv_bfloat16 z = __float2bfloat16(0.f);
        for (int c = threadIdx.x; c < V; c += CE_THREADS) dlogits[r * ldd + c] = z;
      }
    }
    return;
  }
  float m = -INFINITY, s = 0.f;
  if (vec) {
    const __nv_bfloat16* lb = reinterpret_cast<const __nv_bfloat16*>(lr);
    for (int c = threadIdx.x * 8; c < V; c += CE_THREADS * 8) {
      const uint4 u = *reinterpret_cast<const uint4*>(lb + c);
      const float2 a = unpack_bf16(u.x), b2 = unpack_bf16(u.y), c2 = unpack_bf16(u.z), d = unpack_bf16(u.w);
      const float f[8] = {a.x, a.y, b2.x, b2.y, c2.x, c2.y, d.x, d.y};
      float vm = f[0];
#pragma unroll
      for (int j = 1; j < 8; ++j) vm = fmaxf(vm, f[j]);
      if (vm > m) { s *= __expf(m - vm); m = vm; }
#pragma unroll
      for (int j = 0; j < 8; ++j) s += __expf(f[j] - m);
    }
  } else {
    for (int c = threadIdx.x; c < V; c += CE_THREADS) {
      float v = ld_logit<TL>(lr, c);
      if (v > m) { s = s * __expf(m - v) + 1.f; m = v; } else { s += __expf(v - m); }
    }
  }
  const float gm = block_max(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  const float gs = block_sum(s, red);
  const float lse = gm + logf(gs);
  if (threadIdx.x == 0) {
    loss_rows[r] = lse - ld_logit<TL>(lr, label);
    if (lse_rows) lse_rows[r] = lse;
  }
  if (dlogits) {
    const float sc = (grad_scale ? grad_scale[0] : 1.f) * grad_scale_host;
    __syncthreads();  // the label logit has been read before any thread overwrites an aliased buffer
    if (vec) {
      const __nv_bfloat16* lb = reinterpret_cast<const __nv_bfloat16*>(lr);
      constexpr int STEP = CE_THREADS * 8;
      for (int c = (LONG ? (V - 1) / STEP * STEP : 0) + threadIdx.x * 8; LONG ? c >= 0 : c < V; c += LONG ? -STEP : STEP) {
        if (LONG && c >= V) continue;
        const uint4 u = LONG ? __ldcs(reinterpret_cast<const uint4*>(lb + c)) : *reinterpret_cast<const uint4*>(lb + c);
        const float2 a = unpack_bf16(u.x), b2 = unpack_bf16(u.y), c2 = unpack_bf16(u.z), d = unpack_bf16(u.w);
        float f[8] = {a.x, a.y, b2.x, b2.y, c2.x, c2.y, d.x, d.y};
        const int hit = static_cast<int>(label) - c;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float pr = __expf(f[j] - lse);
          if (hit == j) pr -= 1.f;
          f[j] = pr * sc;
        }
        uint4 o;
        o.x = pack_bf16(f[0], f[1]); o.y = pack_bf16(f[2], f[3]); o.z = pack_bf16(f[4], f[5]); o.w = pack_bf16(f[6], f[7]);
        if (LONG) __stcs(reinterpret_cast<uint4*>(dlogits + r * ldd + c), o);
        else *reinterpret_cast<uint4*>(dlogits + r * ldd + c) = o;
      }
    } else {
      for (int c = threadIdx.x; c < V; c += CE_THREADS) {
        float pr = __expf(ld_logit<TL>(lr, c) - lse);
        if (c == label) pr -= 1.f;
        dlogits[r * ldd + c] = __float2bfloat16(pr * sc);
      }
    }
  }
}

// ============================================================================
// out = round(x * g[0]), product in fp32: gradients that a loss formed in its forward, times the gradient of the loss.  Bound by memory: 4096 x
// 151936 bf16 424 us (a copy 380), where torch's conversion, product and conversion back took 3665; 151936 x 2048 fp32 to bf16 1027 -> 305;
// 4096 x 2048 bf16 28 (a product that fetches its factor for each element) -> 12.
// ============================================================================
template <typename TI, typename TO>
__global__ void __launch_bounds__(256)
scale_kernel(const TI* __restrict__ x, const float* __restrict__ g, TO* __restrict__ out, long long n, long long n8) {
  const float f = g[0];
  const long long step = static_cast<long long>(gridDim.x) * 256;
  for (long long q = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x; q < n8; q += step) {
    float v[8];
    if constexpr (sizeof(TI) == 2) {
      load8(reinterpret_cast<const __nv_bfloat16*>(x) + q * 8, v);
    } else {
      const float4 a = reinterpret_cast<const float4*>(x)[2 * q], b = reinterpret_cast<const float4*>(x)[2 * q + 1];
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= f;
    if constexpr (sizeof(TO) == 2) {
      store8(reinterpret_cast<__nv_bfloat16*>(out) + q * 8, v);
    } else {
      reinterpret_cast<float4*>(out)[2 * q] = make_float4(v[0], v[1], v[2], v[3]);
      reinterpret_cast<float4*>(out)[2 * q + 1] = make_float4(v[4], v[5], v[6], v[7]);
    }
  }
  for (long long i = n8 * 8 + static_cast<long long>(blockIdx.x) * 256 + threadIdx.x; i < n; i += step)
    out[i] = static_cast<TO>(static_cast<float>(x[i]) * f);
}

// ============================================================================
// Multi-tensor AdamW on fp32 master shards with optional bf16 shadow copy.
// meta[i] = {p, g, m, v, shadow_bf16 (or 0), numel, g_is_bf16}; chunk table maps
// blockIdx.x -> (tensor, first element).  clip_coef (device scalar, may be null)
// multiplies every gradient; the update is skipped if it is not finite.
// ============================================================================
struct AdamMeta {
  float* p;
  const void* g;
  float* m;
  float* v;
  __nv_bfloat16* shadow;
  long long numel;
  long long g_is_bf16;
};
// 16 K elements per block: with 64 K a replica of 60 M parameters was 920 blocks, less than one full wave, so that SMs with
// one block more than others set the time, and a few hundred thousand parameters used a handful of SMs (310 -> 272 us for the 60 M).
constexpr int ADAM_CHUNK = 16384;

__device__ __forceinline__ void adamw_one(float& p, float g, float& m, float& v, float lr, float beta1, float beta2,
                                          float eps, float decay, float step_size, float bc2_sqrt) {
  p *= decay;
  m = m + (1.f - beta1) * (g - m);
  v = beta2 * v + (1.f - beta2) * g * g;
  p -= step_size * m / (sqrtf(v) / bc2_sqrt + eps);
}

__global__ void __launch_bounds__(256)
adamw_kernel(const AdamMeta* __restrict__ meta, const int2* __restrict__ chunks, float lr, float beta1, float beta2,
             float eps, float weight_decay, float bc1, float bc2_sqrt, const float* __restrict__ clip_coef,
             float grad_prescale) {
  const int2 ch = chunks[blockIdx.x];
  const AdamMeta t = meta[ch.x];
  const long long start = static_cast<long long>(ch.y) * ADAM_CHUNK;
  long long end = start + ADAM_CHUNK;
  if (end > t.numel) end = t.numel;
  float coef = grad_prescale;
  if (clip_coef) {
    float c = clip_coef[0];
    if (!isfinite(c)) return;
    coef *= c;
  }
  const float step_size = lr / bc1;
  const float decay = 1.f - lr * weight_decay;
  const bool aligned = ((reinterpret_cast<uintptr_t>(t.p) | reinterpret_cast<uintptr_t>(t.m) |
                         reinterpret_cast<uintptr_t>(t.v) | reinterpret_cast<uintptr_t>(t.g) |
                         reinterpret_cast<uintptr_t>(t.shadow)) & 15) == 0;
  const long long n4 = aligned ? ((end - start) / 4) : 0;
  for (long long q = threadIdx.x; q < n4; q += blockDim.x) {
    const long long i = start + q * 4;
    float4 p = *reinterpret_cast<const float4*>(t.p + i);
    float4 m = *reinterpret_cast<const float4*>(t.m + i);
    float4 v = *reinterpret_cast<const float4*>(t.v + i);
    float g[4];
    if (t.g_is_bf16) {
      const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(t.g) + i);
      const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
      g[0] = a.x; g[1] = a.y; g[2] = b.x; g[3] = b.y;
    } else {
      const float4 u = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(t.g) + i);
      g[0] = u.x; g[1] = u.y; g[2] = u.z; g[3] = u.w;
    }
    adamw_one(p.x, g[0] * coef, m.x, v.x, lr, beta1, beta2, eps, decay, step_size, bc2_sqrt);
    adamw_one(p.y, g[1] * coef, m.y, v.y, lr, beta1, beta2, eps, decay, step_size, bc2_sqrt);
    adamw_one(p.z, g[2] * coef, m.z, v.z, lr, beta1, beta2, eps, decay, step_size, bc2_sqrt);
    adamw_one(p.w, g[3] * coef, m.w, v.w, lr, beta1, beta2, eps, decay, step_size, bc2_sqrt);
    *reinterpret_cast<float4*>(t.p + i) = p;
    *reinterpret_cast<float4*>(t.m + i) = m;
    *reinterpret_cast<float4*>(t.v + i) = v;
    if (t.shadow) {
      uint2 o;
      o.x = pack_bf16(p.x, p.y); o.y = pack_bf16(p.z, p.w);
      *reinterpret_cast<uint2*>(t.shadow + i) = o;
    }
  }
  for (long long i = start + n4 * 4 + threadIdx.x; i < end; i += blockDim.x) {
    float g = t.g_is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(t.g)[i])
                          : reinterpret_cast<const float*>(t.g)[i];
    float p = t.p[i], m = t.m[i], v = t.v[i];
    adamw_one(p, g * coef, m, v, lr, beta1, beta2, eps, decay, step_size, bc2_sqrt);
    t.p[i] = p; t.m[i] = m; t.v[i] = v;
    if (t.shadow) t.shadow[i] = __float2bfloat16(p);
  }
}

// Squared-norm partials: partial[blockIdx.x] = sum over the chunk of g^2 (fp32).
__global__ void __launch_bounds__(256)
sqnorm_kernel(const AdamMeta* __restrict__ meta, const int2* __restrict__ chunks, float* __restrict__ partial,
              float prescale) {
  __shared__ float red[32];
  const int2 ch = chunks[blockIdx.x];
  const AdamMeta t = meta[ch.x];
  const long long start = static_cast<long long>(ch.y) * ADAM_CHUNK;
  long long end = start + ADAM_CHUNK;
  if (end > t.numel) end = t.numel;
  float s = 0.f;
  const bool aligned = (reinterpret_cast<uintptr_t>(t.g) & 15) == 0;
  // Sixteen bytes a load, and four loads of a thread on their way at a time: fp32 gradients, which went by single
  // words, 72 -> 53 us for 60 M and 328 -> 238 us (6.7 TB/s) for 400 M; bf16 ones had their 16 bytes before (35 and 137 us).
  long long done = 0;
  if (aligned && t.g_is_bf16) {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(t.g) + start);
    const int n8 = static_cast<int>((end - start) / 8);
#pragma unroll 4
    for (int q = threadIdx.x; q < n8; q += 256) {
      const uint4 u = __ldg(src + q);
      const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
      s += a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y + c.x * c.x + c.y * c.y + d.x * d.x + d.y * d.y;
    }
    done = static_cast<long long>(n8) * 8;
  } else if (aligned) {
    const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(t.g) + start);
    const int n4 = static_cast<int>((end - start) / 4);
#pragma unroll 4
    for (int q = threadIdx.x; q < n4; q += 256) {
      const float4 u = __ldg(src + q);
      s += u.x * u.x + u.y * u.y + u.z * u.z + u.w * u.w;
    }
    done = static_cast<long long>(n4) * 4;
  }
  for (long long i = start + done + threadIdx.x; i < end; i += 256) {
    float g = t.g_is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(t.g)[i])
                          : reinterpret_cast<const float*>(t.g)[i];
    s += g * g;
  }
  s = block_sum(s, red) * prescale * prescale;
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// Words between the device and pinned host memory, which the kernel reads or writes where it lies: one launch in line with its neighbours.
// The copy engine in its place hands the stream over and back: an optimizer step on 60 M parameters, which has one copy each way, took
// 347 us with it and takes 337.
__global__ void __launch_bounds__(256) words_kernel(int* __restrict__ dst, const int* __restrict__ src, long long n) {
  for (long long i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) dst[i] = src[i];
}

// out[0] = sum(partial[0..n)) + extra_sq ; out[1] = sqrt(out[0]) ; out[2] = min(1, max_norm/(norm+1e-6))
__global__ void clip_coef_kernel(const float* __restrict__ partial, int n, const float* __restrict__ extra_sq,
                                 float max_norm, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) {
    if (extra_sq) s += extra_sq[0];
    float norm = sqrtf(s);
    out[0] = s;
    out[1] = norm;
    float c = max_norm / (norm + 1e-6f);
    out[2] = (max_norm > 0.f) ? fminf(c, 1.f) : 1.f;
    if (!isfinite(norm)) out[2] = norm;  // propagates NaN/Inf so the update is skipped
  }
}

}  // namespace ttb

// ----------------------------------------------------------------------------
// C ABI
// ----------------------------------------------------------------------------
using namespace ttb;
#define STREAM(s) reinterpret_cast<cudaStream_t>(s)
#define LAUNCH_RET() do { cudaError_t e__ = cudaGetLastError(); return e__ == cudaSuccess ? 0 : 400 + (int)e__; } while (0)

TTB_EXPORT int ttb_rmsnorm_fwd(const void* x, const void* residual, const void* w, void* y, void* sum_out,
                               float* rstd, long long T, int H, float eps, int one_plus_w, void* stream) {
  if (H % 8) return 901;
  if (T == 0) return 0;
  int threads = H / 8;
  threads = threads > 256 ? 256 : ((threads + 31) / 32) * 32;
  const int iters = (H + threads * 8 - 1) / (threads * 8);
  auto X = (const __nv_bfloat16*)x; auto R = (const __nv_bfloat16*)residual; auto W = (const __nv_bfloat16*)w;
  if (iters <= 1) rmsnorm_fwd_kernel<1><<<(unsigned)T, threads, 0, STREAM(stream)>>>(X, R, W, (__nv_bfloat16*)y, (__nv_bfloat16*)sum_out, rstd, H, eps, one_plus_w);
  else if (iters <= 4) rmsnorm_fwd_kernel<4><<<(unsigned)T, threads, 0, STREAM(stream)>>>(X, R, W, (__nv_bfloat16*)y, (__nv_bfloat16*)sum_out, rstd, H, eps, one_plus_w);
  else return 902;
  LAUNCH_RET();
}

// dw_partial must hold grid*H floats; returns the grid size used through *grid_out.
TTB_EXPORT int ttb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres_in,
                               void* dx, float* dw_partial, void* dw_out, int dw_bf16, long long T, int H, int one_plus_w,
                               int grid, void* stream) {
  if (H % 8) return 901;
  if (T == 0) return 0;
  if (H > 8192) return 902;
  const RowPlan plan = row_plan(T, H, grid);
  grid = plan.grid;
  auto DY = (const __nv_bfloat16*)dy; auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w;
  ROW_KERNEL(rmsnorm_bwd_kernel, plan)<<<grid, plan.threads, 0, STREAM(stream)>>>(
      DY, X, W, rstd, (const __nv_bfloat16*)dres_in, (__nv_bfloat16*)dx, dw_partial, T, H, one_plus_w);
  colsum(dw_partial, dw_out, dw_bf16, grid, H, STREAM(stream));
  LAUNCH_RET();
}

TTB_EXPORT int ttb_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd,
                                 long long T, int H, float eps, void* stream) {
  if (H % 8) return 901;
  if (T == 0) return 0;
  int threads = H / 8;
  threads = threads > 256 ? 256 : ((threads + 31) / 32) * 32;
  const int iters = (H + threads * 8 - 1) / (threads * 8);
  auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w; auto B = (const __nv_bfloat16*)b;
  if (iters <= 1) layernorm_fwd_kernel<1><<<(unsigned)T, threads, 0, STREAM(stream)>>>(X, W, B, (__nv_bfloat16*)y, mean, rstd, H, eps);
  else if (iters <= 4) layernorm_fwd_kernel<4><<<(unsigned)T, threads, 0, STREAM(stream)>>>(X, W, B, (__nv_bfloat16*)y, mean, rstd, H, eps);
  else return 902;
  LAUNCH_RET();
}

// part must hold grid * 2 * H floats; dwdb_out receives [2][H] (dw then db).
TTB_EXPORT int ttb_layernorm_bwd(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, void* dx,
                                 float* part, void* dwdb_out, int out_bf16, long long T, int H, int grid, void* stream) {
  if (H % 8) return 901;
  if (T == 0) return 0;
  if (H > 8192) return 902;
  const RowPlan plan = row_plan(T, H, grid);
  grid = plan.grid;
  auto DY = (const __nv_bfloat16*)dy; auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w;
  ROW_KERNEL(layernorm_bwd_kernel, plan)<<<grid, plan.threads, 0, STREAM(stream)>>>(DY, X, W, mean, rstd,
                                                                                                       (__nv_bfloat16*)dx, part, T, H);
  colsum(part, dwdb_out, out_bf16, grid, 2 * H, STREAM(stream));
  LAUNCH_RET();
}

// x, y on 8-byte boundaries, strides multiples of 4 elements; cos / sin fp32 [T, half] on 16-byte boundaries
TTB_EXPORT int ttb_rope(const void* x, long long x_t, long long x_h, const float* cos_t, const float* sin_t, void* y, long long T,
                        int heads, int half, float sign, void* stream) {
  if (half % 4 || x_t % 4 || x_h % 4) return 901;
  if (((uintptr_t)x | (uintptr_t)y) & 7 || ((uintptr_t)cos_t | (uintptr_t)sin_t) & 15) return 902;
  const long long total = T * heads * (half / 4);
  if (total == 0) return 0;
  rope_kernel<<<(unsigned)((total + 255) / 256), 256, 0, STREAM(stream)>>>((const __nv_bfloat16*)x, x_t, x_h, cos_t, sin_t,
                                                                          (__nv_bfloat16*)y, total, heads, half, sign);
  LAUNCH_RET();
}

template <bool BACK>
static int qkv_rope(const void* x, const void* bias, const float* cos_t, const float* sin_t, void* q, void* k, void* v, void* dx, float* part,
                    long long T, int heads, int half, int grid, cudaStream_t stream) {
  if (half < 4 || half % 4 || heads < 1) return 901;
  if (((uintptr_t)x | (uintptr_t)bias | (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)dx) & 7 || ((uintptr_t)cos_t | (uintptr_t)sin_t | (uintptr_t)part) & 15)
    return 902;
  const long long groups = 3LL * heads * (half / 4);
  if (groups > 4 * 512) return 903;
  const int items = groups <= 512 ? 1 : groups <= 1024 ? 2 : 4;
  const int threads = static_cast<int>(((groups + items - 1) / items + 31) / 32 * 32);
  auto run = [&](auto kernel) {
    kernel<<<grid, threads, 0, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)bias, cos_t, sin_t, (__nv_bfloat16*)q, (__nv_bfloat16*)k,
                                         (__nv_bfloat16*)v, (__nv_bfloat16*)dx, part, T, heads, half);
  };
  if (items == 1) run(qkv_rope_kernel<1, BACK>);
  else if (items == 2) run(qkv_rope_kernel<2, BACK>);
  else run(qkv_rope_kernel<4, BACK>);
  return 0;
}

// x, bias, q, k, v: bf16 on 8-byte boundaries, contiguous; cos / sin fp32 [T, half] on 16-byte boundaries; 3 heads half / 4 <= 2048
TTB_EXPORT int ttb_qkv_rope_fwd(const void* x, const void* bias, const float* cos_t, const float* sin_t, void* q, void* k, void* v, long long T,
                                int heads, int half, int grid, void* stream) {
  if (T == 0) return 0;
  if (int e = qkv_rope<false>(x, bias, cos_t, sin_t, q, k, v, nullptr, nullptr, T, heads, half, grid, STREAM(stream))) return e;
  LAUNCH_RET();
}

// part: fp32 [grid, 6 heads half]; dbias: a row's width, fp32 or bf16
TTB_EXPORT int ttb_qkv_rope_bwd(const void* dq, const void* dk, const void* dv, const float* cos_t, const float* sin_t, void* dx, float* part,
                                void* dbias, int out_bf16, long long T, int heads, int half, int grid, void* stream) {
  if (T == 0) return 0;
  if (int e = qkv_rope<true>(nullptr, nullptr, cos_t, sin_t, const_cast<void*>(dq), const_cast<void*>(dk), const_cast<void*>(dv), dx, part, T, heads,
                             half, grid, STREAM(stream)))
    return e;
  colsum(part, dbias, out_bf16, grid, 6 * heads * half, STREAM(stream));
  LAUNCH_RET();
}

TTB_EXPORT int ttb_bias_act_fwd(const void* x, const void* bias, const void* residual, void* y, long long R, int C, int act,
                                void* stream) {
  if (C % 8 || act < 0 || act > 2) return 901;
  if (R == 0) return 0;
  const long long total = R * (C / 8);
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  bias_act_fwd_kernel<<<(unsigned)blocks, 256, 0, STREAM(stream)>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)bias,
                                                                    (const __nv_bfloat16*)residual, (__nv_bfloat16*)y, R, C, act);
  LAUNCH_RET();
}

// part must hold grid * C floats; dx may be null (identity activation: d(x) is dy itself).
TTB_EXPORT int ttb_bias_act_bwd(const void* dy, const void* x, const void* bias, void* dx, float* part, void* dbias_out, int out_bf16,
                                long long R, int C, int act, int grid, void* stream) {
  if (C % 8 || act < 0 || act > 2) return 901;
  if (R == 0) return 0;
  if (C > 16384) return 902;
  if (grid > R) grid = (int)R;
  const int threads = row_threads(C > 8192 ? (C + 15) / 16 * 8 : C);
  bias_act_bwd_kernel<<<dim3(grid, C > 8192 ? 2 : 1), threads, 0, STREAM(stream)>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,
                                                                                 (const __nv_bfloat16*)bias, (__nv_bfloat16*)dx, part, R, C, act);
  colsum(part, dbias_out, out_bf16, grid, C, STREAM(stream));
  LAUNCH_RET();
}

// A thread owns 4 channels of a filter of up to four taps, else 8.  Blocks per SM: up to four taps, whole waves of what an SM holds, one
// of the backward (4; its rows of overlap and column sums grow with the number of blocks: 8, 12 and 24 per SM take 85, 91 and 109 us
// against 79) and two of the forward (12; 41 us, one wave 42, and 100 against 104 us for 16384 x 6144).  Where two waves of the forward
// leave a block less than 14 rows, of which three more are read before the first, it is one wave of whole steps of four rows, and fewer
// rows only where there would not be a block for every SM.  Two waves -> this, inputs from memory: 4096 x 512 7.7 -> 6.2 us, 300 x 8192
// 8.5 -> 6.8, 2047 x 1024 7.8 -> 6.1, 1001 x 3072 8.4 -> 7.5, 64 x 12288 6.9 -> 3.8, 16 x 512 2.0 (two rows a block 2.2); 15 rows with two
// waves 17.4 (2047 x 6144), with one 17.8.
static void conv_grid(long long T, int D, int W, bool bwd, int& threads, dim3& grid, int& rows_per_block) {
  const int vec = W <= 4 ? D / 4 : D / 8;
  threads = vec >= 128 ? 128 : ((vec + 31) / 32) * 32;
  const int gx = (vec + threads - 1) / threads;
  const long long sms = device_sms();
  long long want = W <= 4 ? sms * (bwd ? 4 : 12) / gx : (sms * 8 + gx - 1) / gx;
  if (want > T) want = T;
  if (want < 1) want = 1;
  rows_per_block = static_cast<int>((T + want - 1) / want);
  if (W <= 4 && !bwd && rows_per_block < 14) {
    const long long steps = (T * gx + sms * 6 * CONV_ROWS - 1) / (sms * 6 * CONV_ROWS), each = (T * gx + sms - 1) / sms;
    rows_per_block = static_cast<int>(steps * CONV_ROWS < each ? steps * CONV_ROWS : each);
  }
  grid = dim3(gx, static_cast<unsigned>((T + rows_per_block - 1) / rows_per_block));
}

TTB_EXPORT int ttb_causal_conv1d_fwd(const void* x, const void* w, const void* bias, const int* seq_start, void* y,
                                     long long T, int D, int W, int silu, void* stream) {
  if (D % 8 || W < 1 || W > CONV_MAX_W) return 901;
  if (T == 0) return 0;
  int threads, rpb;
  dim3 grid;
  conv_grid(T, D, W, false, threads, grid, rpb);
  if (W <= 4)
    causal_conv1d_w4_kernel<false><<<grid, threads, 0, STREAM(stream)>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
        (const __nv_bfloat16*)bias, seq_start, nullptr, (__nv_bfloat16*)y, nullptr, T, D, W, silu, rpb);
  else
    causal_conv1d_kernel<false, 8><<<grid, threads, 0, STREAM(stream)>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
        (const __nv_bfloat16*)bias, seq_start, nullptr, (__nv_bfloat16*)y, nullptr, T, D, W, silu, rpb);
  LAUNCH_RET();
}

// part must hold row_blocks * (W + 1) * D floats (row_blocks from ttb_causal_conv1d_row_blocks); dwdb_out: [(W + 1), D]
TTB_EXPORT int ttb_causal_conv1d_row_blocks(long long T, int D, int W) {
  int threads, rpb;
  dim3 grid;
  conv_grid(T > 0 ? T : 1, D, W, true, threads, grid, rpb);
  return static_cast<int>(grid.y);
}

TTB_EXPORT int ttb_causal_conv1d_bwd(const void* dy, const void* x, const void* w, const void* bias, const int* seq_start,
                                     const int* seq_end, void* dpre /* W > 4 only */, void* dx, float* part, float* dwdb_out, long long T,
                                     int D, int W, int silu, void* stream) {
  if (D % 8 || W < 1 || W > CONV_MAX_W) return 901;
  if (T == 0) return 0;
  int threads, rpb;
  dim3 grid;
  conv_grid(T, D, W, true, threads, grid, rpb);
  if (W <= 4) {
    causal_conv1d_w4_kernel<true><<<grid, threads, 0, STREAM(stream)>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
        (const __nv_bfloat16*)bias, seq_start, (const __nv_bfloat16*)dy, (__nv_bfloat16*)dx, part, T, D, W, silu, rpb);
  } else {
    causal_conv1d_kernel<true, 8><<<grid, threads, 0, STREAM(stream)>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
        (const __nv_bfloat16*)bias, seq_start, (const __nv_bfloat16*)dy, (__nv_bfloat16*)dpre, part, T, D, W, silu, rpb);
    causal_conv1d_dx_kernel<8><<<grid, threads, 0, STREAM(stream)>>>((const __nv_bfloat16*)dpre, (const __nv_bfloat16*)w,
                                                                     seq_end, (__nv_bfloat16*)dx, T, D, W, rpb);
  }
  const int cols = (W + 1) * D;
  colsum(part, dwdb_out, 0, static_cast<int>(grid.y), cols, STREAM(stream));
  LAUNCH_RET();
}

TTB_EXPORT int ttb_qknorm_rope_fwd(const void* qkv, long long ld, int Hq, int Hk, int D, const void* wq, const void* wk,
                                   const float* cos_t, const float* sin_t, void* q_out, void* k_out, float* rstd,
                                   long long T, float eps, int use_norm, void* stream) {
  if (D != 128) return 901;
  if (((uintptr_t)qkv | (uintptr_t)q_out | (uintptr_t)k_out | (uintptr_t)wq | (uintptr_t)wk) & 7 || ld % 4) return 902;
  if (((uintptr_t)cos_t | (uintptr_t)sin_t) & 15) return 902;
  const long long items = T * (Hq + Hk);
  if (items == 0) return 0;
  const long long blocks = (items + 15) / 16;
  qknorm_rope_fwd_kernel<<<(unsigned)blocks, 256, 0, STREAM(stream)>>>(
      (const __nv_bfloat16*)qkv, ld, Hq, Hk, (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, cos_t, sin_t,
      (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_out, rstd, T, eps, use_norm);
  LAUNCH_RET();
}

// dv (optional, [T, Hk, 128] contiguous) goes to the v columns of dqkv.  With use_norm: part holds grid * 256 floats, dw_out
// [2, 128] (dwq, dwk) in fp32 or bf16.
TTB_EXPORT int ttb_qknorm_rope_bwd(const void* dq, const void* dk, const void* dv, const void* qkv, long long ld, int Hq, int Hk, int D,
                                   const void* wq, const void* wk, const float* cos_t, const float* sin_t,
                                   const float* rstd, void* dqkv, long long ldd, float* part, void* dw_out, int dw_bf16, long long T,
                                   int use_norm, int grid, void* stream) {
  if (D != 128) return 901;
  if (T == 0) return 0;
  qknorm_rope_bwd_kernel<<<grid, 256, 0, STREAM(stream)>>>(
      (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, (const __nv_bfloat16*)qkv, ld, Hq, Hk,
      (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, cos_t, sin_t, rstd, (__nv_bfloat16*)dqkv, ldd, part, T, use_norm);
  if (use_norm) colsum(part, dw_out, dw_bf16, grid, 2 * 128, STREAM(stream));
  LAUNCH_RET();
}

TTB_EXPORT int ttb_swiglu_fwd(const void* x, long long ldx, void* y, long long ldy, const float* row_scale, long long R,
                              int F, const int* nrows, void* stream) {
  if (F % 8 || ldx % 8 || ldy % 8) return 901;
  const long long n = R * F / 8;
  if (n == 0) return 0;
  swiglu_fwd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, STREAM(stream)>>>((const __nv_bfloat16*)x, ldx,
                                                                            (__nv_bfloat16*)y, ldy, row_scale, R, F, nrows);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_swiglu_bwd(const void* dy, long long lddy, const void* x, long long ldx, const float* row_scale,
                              void* dx, long long lddx, float* dscale, void* y_out, long long ldy, long long R, int F,
                              const int* nrows, void* stream) {
  if (F % 8 || ldx % 8 || lddy % 8 || lddx % 8 || (y_out && ldy % 8)) return 901;
  if (R == 0) return 0;
  int threads = F / 8;
  threads = threads > 256 ? 256 : ((threads + 31) / 32) * 32;
  swiglu_bwd_kernel<<<(unsigned)R, threads, 0, STREAM(stream)>>>((const __nv_bfloat16*)dy, lddy,
                                                                (const __nv_bfloat16*)x, ldx, row_scale,
                                                                (__nv_bfloat16*)dx, lddx, dscale, (__nv_bfloat16*)y_out, ldy, F, nrows);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_cross_entropy(const void* logits, int logits_fp32, long long ldl, const long long* labels,
                                 float* loss_rows, float* lse_rows, void* dlogits, long long ldd,
                                 const float* grad_scale, float grad_scale_host, long long R, int V, void* stream) {
  if (R == 0) return 0;
  auto run = [&](auto kernel, auto* rows) {
    kernel<<<(unsigned)R, CE_THREADS, 0, STREAM(stream)>>>(rows, ldl, labels, loss_rows, lse_rows, (__nv_bfloat16*)dlogits, ldd, grad_scale,
                                                           grad_scale_host, V);
  };
  if (logits_fp32) run(cross_entropy_kernel<float, false>, (const float*)logits);
  else if (ce_long(V, dlogits == logits)) run(cross_entropy_kernel<__nv_bfloat16, true>, (const __nv_bfloat16*)logits);
  else run(cross_entropy_kernel<__nv_bfloat16, false>, (const __nv_bfloat16*)logits);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_adam_chunk_elems() { return ADAM_CHUNK; }

TTB_EXPORT int ttb_adamw(const void* meta, const void* chunks, int n_chunks, float lr, float beta1, float beta2,
                         float eps, float weight_decay, float bc1, float bc2_sqrt, const float* clip_coef,
                         float grad_prescale, void* stream) {
  if (n_chunks == 0) return 0;
  adamw_kernel<<<n_chunks, 256, 0, STREAM(stream)>>>((const AdamMeta*)meta, (const int2*)chunks, lr, beta1, beta2, eps,
                                                     weight_decay, bc1, bc2_sqrt, clip_coef, grad_prescale);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_grad_sqnorm(const void* meta, const void* chunks, int n_chunks, float* partial, float prescale,
                               void* stream) {
  if (n_chunks == 0) return 0;
  sqnorm_kernel<<<n_chunks, 256, 0, STREAM(stream)>>>((const AdamMeta*)meta, (const int2*)chunks, partial, prescale);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_scale(const void* x, int x_bf16, const float* g, void* out, int out_bf16, long long n, int num_sms, void* stream) {
  if (n <= 0) return 0;
  const long long n8 = (((uintptr_t)x | (uintptr_t)out) & 15) ? 0 : n / 8;
  const long long need = ((n8 ? n8 : n) + 255) / 256;
  const int grid = static_cast<int>(need < 8LL * num_sms ? need : 8LL * num_sms);
  auto run = [&](auto* src, auto* dst) { scale_kernel<<<grid, 256, 0, STREAM(stream)>>>(src, g, dst, n, n8); };
  auto xb = (const __nv_bfloat16*)x; auto xf = (const float*)x; auto ob = (__nv_bfloat16*)out; auto of = (float*)out;
  if (x_bf16 && out_bf16) run(xb, ob);
  else if (x_bf16) run(xb, of);
  else if (out_bf16) run(xf, ob);
  else run(xf, of);
  LAUNCH_RET();
}

// n 32-bit words; either side may be pinned host memory
TTB_EXPORT int ttb_copy_words(void* dst, const void* src, long long n, void* stream) {
  if (n <= 0) return 0;
  words_kernel<<<static_cast<int>(n > 64 * 256 ? 64 : (n + 255) / 256), 256, 0, STREAM(stream)>>>((int*)dst, (const int*)src, n);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_clip_coef(const float* partial, int n, const float* extra_sq, float max_norm, float* out3,
                             void* stream) {
  clip_coef_kernel<<<1, 1024, 0, STREAM(stream)>>>(partial, n, extra_sq, max_norm, out3);
  LAUNCH_RET();
}

// ----------------------------------------------------------------------------
// Allocation-free RMSNorm backward (see ttb_noalloc.h for the contract).
// The scratch that ttb_rmsnorm_bwd receives from its caller lives here in a file-scope device array.  In host code
// the name `g_noalloc_scratch` is only a handle for the runtime; the address a kernel can use comes from
// cudaGetSymbolAddress, looked up once per device with that device current.
// ----------------------------------------------------------------------------
#include "ttb_noalloc.h"

static __device__ __align__(256) float g_noalloc_scratch[TTB_NOALLOC_BLOCKS * TTB_NOALLOC_MAX_H];

namespace {
constexpr int kMaxDevices = 64;
float* g_noalloc_ptr[kMaxDevices] = {nullptr};

// Device address of the scratch array on the current device (cached).  Returns 0 or a TTB_NOALLOC_ERR_SYMBOL code.
int noalloc_scratch(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) return TTB_NOALLOC_ERR_SYMBOL + static_cast<int>(e);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) return TTB_NOALLOC_ERR_SYMBOL + static_cast<int>(e);
    g_noalloc_ptr[dev] = static_cast<float*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}
}  // namespace

TTB_EXPORT int ttb_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w, const float* rstd,
                                       const void* dres_in, void* dx, float* dw_out, long long T, int H,
                                       int one_plus_w, void* stream) {
  if (H <= 0 || (H % 8) != 0 || H > TTB_NOALLOC_MAX_H || T < 0) return TTB_NOALLOC_ERR_SIZE;
  if (T == 0) return TTB_NOALLOC_OK;
  float* scratch = nullptr;
  const int rc = noalloc_scratch(&scratch);
  if (rc != 0) return rc;
  const RowPlan plan = row_plan(T, H, TTB_NOALLOC_BLOCKS);
  const int grid = plan.grid;
  auto DY = (const __nv_bfloat16*)dy; auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w;
  // every block writes its full row of `scratch` (H floats), and the column sum below reads exactly rows [0, grid):
  // nothing has to be cleared between calls
  ROW_KERNEL(rmsnorm_bwd_kernel, plan)<<<grid, plan.threads, 0, STREAM(stream)>>>(
      DY, X, W, rstd, (const __nv_bfloat16*)dres_in, (__nv_bfloat16*)dx, scratch, T, H, one_plus_w);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return TTB_NOALLOC_ERR_LAUNCH_DX + static_cast<int>(e);
  colsum(scratch, dw_out, 0, grid, H, STREAM(stream));
  e = cudaGetLastError();
  return e == cudaSuccess ? TTB_NOALLOC_OK : TTB_NOALLOC_ERR_LAUNCH_DW + static_cast<int>(e);
}

TTB_EXPORT const char* ttb_noalloc_strerror(int code) {
  if (code == TTB_NOALLOC_OK) return "ok";
  if (code == TTB_NOALLOC_ERR_SIZE)
    return "ttb_rmsnorm_bwd_noalloc: H must be a positive multiple of 8 and at most 8192 (TTB_NOALLOC_MAX_H), T >= 0";
  if (code >= TTB_NOALLOC_ERR_SYMBOL && code < TTB_NOALLOC_ERR_SYMBOL + 10000)
    return "ttb_rmsnorm_bwd_noalloc: could not resolve the device address of the built-in scratch array "
           "(cudaGetDevice / cudaGetSymbolAddress failed; code - 200000 is the CUDA error)";
  if (code >= TTB_NOALLOC_ERR_LAUNCH_DW && code < TTB_NOALLOC_ERR_LAUNCH_DW + 10000)
    return "ttb_rmsnorm_bwd_noalloc: launch of the weight-gradient column sum failed (code - 110000 is the CUDA error)";
  if (code >= TTB_NOALLOC_ERR_LAUNCH_DX && code < TTB_NOALLOC_ERR_LAUNCH_DX + 10000)
    return "ttb_rmsnorm_bwd_noalloc: launch of the dx / partial-sum kernel failed (code - 100000 is the CUDA error)";
  return "ttb_rmsnorm_bwd_noalloc: unknown error code";
}
