// Kernels of the delta rule with one decay per head and key channel (Kimi delta attention).  Formulas and arithmetic as in
// delta_chunk.cuh with D_ij,c = exp(G_ic - G_jc) inside every sum over channels c:
//
//   L_ij = beta_i sum_c k^_ic k^_jc D_ij,c          A_ij = sum_c q^_ic k^_jc D_ij,c
//
// Those sums do not factor into a matrix product without exponents of either sign (e^G_i and e^-G_j overflow together), so
// they are evaluated pair by pair, 266 k exponentials per chunk and head and direction: about 9 us of the special function
// units of one SM, against which the products with the states run on the tensor cores as before.  All other decays are
// products of two non-positive exponents of one row.  G is kept in units of log2, so that a decay is one subtraction and
// one exp2.
//
// The backward is split in two so that each half fits one SM's shared memory: `score` (T^T dx, dL, dA and the pairwise
// sums) and `state` (products with S and dS, and the final gradients); 128 KB per chunk and head pass between them.
//
// Measured (2047 tokens, 8 heads, three documents): prep 54 us, out 42, bwd_pre 22, score 92, state 73; the operator with its
// gates, forward + backward, takes 0.86 ms (6.9 ms and 467 launches as batched torch products, 21 launches now).
#include "delta_chunk.cuh"

namespace ttb {

constexpr int DV_G = 132;    // row stride of G and of tiles read down their columns
constexpr int DV_A = 136;    // row stride of fp32 tiles read in pairs along a row

// G (units of log2) of a chunk: cumulative sums down 64 rows for 128 channels.  Starts without, ends with a barrier, which also
// publishes the tiles that this thread block has asked for before.
template <int NT>
__device__ __forceinline__ void dv_cumsum(const DeltaChunkIn& p, float* sG, int ld, int row0, int n, int h) {
  constexpr int PARTS = NT / 128, ROWS = 64 / PARTS;
  const int c = threadIdx.x & 127, part = threadIdx.x >> 7;
  const float* src = p.g + (static_cast<long long>(row0) * p.H + h) * DC_D + c;
  const long long step = static_cast<long long>(p.H) * DC_D;
  float v[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) v[r] = part * ROWS + r < n ? __ldg(src + (part * ROWS + r) * step) : 0.f;
  dc_wait();
  float run = 0.f;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    run += v[r] * 1.44269504f;
    v[r] = run;
  }
  sG[(part * ROWS + ROWS - 1) * ld + c] = run;
  __syncthreads();
  float before = 0.f;
#pragma unroll
  for (int q = 0; q < PARTS - 1; ++q)
    if (q < part) before += sG[(q * ROWS + ROWS - 1) * ld + c];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ROWS; ++r) sG[(part * ROWS + r) * ld + c] = v[r] + before;
  __syncthreads();
}
__device__ __forceinline__ float4 dv_bf4(const __nv_bfloat16* s) {
  const uint2 u = *reinterpret_cast<const uint2*>(s);
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}

// ------------------------------------------------------------------------------------------------
// prep
// ------------------------------------------------------------------------------------------------
struct VpSmem {
  static constexpr int QV = 0, K = QV + DC_C * DC_QS * 2, G = K + DC_C * DC_QS * 2;
  static constexpr int L = G + DC_C * DV_G * 4, T = L + DC_C * DP_LT * 4, ROWS = T + DC_C * DP_LT * 4;
  static constexpr int TOTAL = ROWS + 3 * DC_C * 4 + DC_D * 4;
};

__global__ void __launch_bounds__(256, 2)
delta_vec_prep_kernel(const DeltaChunkIn p, float* __restrict__ Tg, float* __restrict__ Ag, float* __restrict__ U,
                      __nv_bfloat16* __restrict__ W, __nv_bfloat16* __restrict__ Ko, float* __restrict__ decay) {
  extern __shared__ __align__(16) uint8_t sm[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(sm + VpSmem::QV);   // q, later v
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(sm + VpSmem::K);
  float* sG = reinterpret_cast<float*>(sm + VpSmem::G);                     // G, later beta k^ e^G
  float* sL = reinterpret_cast<float*>(sm + VpSmem::L);
  float* sT = reinterpret_cast<float*>(sm + VpSmem::T);
  float* sB = reinterpret_cast<float*>(sm + VpSmem::ROWS);
  float *sRk = sB + DC_C, *sRq = sRk + DC_C, *sGL = sRq + DC_C;
  const int c = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1];
  const long long hc = static_cast<long long>(h) * p.NC + c;
  dc_load_rows<256>(sQ, p.q + row0 * p.q_t + h * p.q_h, p.q_t, n);
  dc_load_rows<256>(sK, p.k + row0 * p.k_t + h * p.k_h, p.k_t, n);
  if (tid < DC_C) sB[tid] = tid < n ? __ldg(p.beta + static_cast<long long>(row0 + tid) * p.H + h) : 0.f;
  dv_cumsum<256>(p, sG, DV_G, row0, n, h);
  dc_row_norms<256>(sQ, sRq, p.scale, sK, sRk, 1.f, p.l2);
  if (tid < DC_D) {
    const float gl = sG[(DC_C - 1) * DV_G + tid];
    sGL[tid] = gl;
    decay[hc * DC_D + tid] = exp2f(gl);
  }
  __syncthreads();
  float* Aout = Ag + hc * DC_C * DC_C;
  for (int e = tid; e < DC_C * DC_C; e += 256) {
    const int i = e >> 6, j = e & 63;
    if (j >= i) sL[i * DP_LT + j] = 0.f;
    if (j > i) Aout[e] = 0.f;
  }
  // ---- pairwise scores: 2 x 2 pairs per thread below the diagonal (496 tiles, two rounds of 248 threads) ...
  for (int t = tid; t < 496 && tid < 248; t += 248) {
    int bi = static_cast<int>((1.f + sqrtf(1.f + 8.f * t)) * 0.5f);
    while (bi * (bi - 1) / 2 > t) --bi;
    while ((bi + 1) * bi / 2 <= t) ++bi;
    const int i = 2 * bi, j = 2 * (t - bi * (bi - 1) / 2);
    float ak[2][2] = {}, aq[2][2] = {};
#pragma unroll 2
    for (int ch = 0; ch < DC_D; ch += 4) {
      const float4 gi[2] = {*reinterpret_cast<const float4*>(sG + i * DV_G + ch), *reinterpret_cast<const float4*>(sG + (i + 1) * DV_G + ch)};
      const float4 gj[2] = {*reinterpret_cast<const float4*>(sG + j * DV_G + ch), *reinterpret_cast<const float4*>(sG + (j + 1) * DV_G + ch)};
      const float4 ki[2] = {dv_bf4(sK + i * DC_QS + ch), dv_bf4(sK + (i + 1) * DC_QS + ch)};
      const float4 qi[2] = {dv_bf4(sQ + i * DC_QS + ch), dv_bf4(sQ + (i + 1) * DC_QS + ch)};
      const float4 kj[2] = {dv_bf4(sK + j * DC_QS + ch), dv_bf4(sK + (j + 1) * DC_QS + ch)};
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const float t0 = exp2f(gi[a].x - gj[b].x) * kj[b].x, t1 = exp2f(gi[a].y - gj[b].y) * kj[b].y;
          const float t2 = exp2f(gi[a].z - gj[b].z) * kj[b].z, t3 = exp2f(gi[a].w - gj[b].w) * kj[b].w;
          ak[a][b] = fmaf(ki[a].x, t0, fmaf(ki[a].y, t1, fmaf(ki[a].z, t2, fmaf(ki[a].w, t3, ak[a][b]))));
          aq[a][b] = fmaf(qi[a].x, t0, fmaf(qi[a].y, t1, fmaf(qi[a].z, t2, fmaf(qi[a].w, t3, aq[a][b]))));
        }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const float rk = sB[i + a] * sRk[i + a], rq = sRq[i + a];
      *reinterpret_cast<float2*>(sL + (i + a) * DP_LT + j) = make_float2(ak[a][0] * (rk * sRk[j]), ak[a][1] * (rk * sRk[j + 1]));
      *reinterpret_cast<float2*>(Aout + (i + a) * DC_C + j) = make_float2(aq[a][0] * (rq * sRk[j]), aq[a][1] * (rq * sRk[j + 1]));
    }
  }
  {
    // ... and the 32 tiles on the diagonal, eight threads each
    const int i = (tid >> 3) * 2, c0 = (tid & 7) * 16;
    float q00 = 0.f, q11 = 0.f, q10 = 0.f, k10 = 0.f;
#pragma unroll
    for (int ch = c0; ch < c0 + 16; ch += 4) {
      const float4 g0 = *reinterpret_cast<const float4*>(sG + i * DV_G + ch), g1 = *reinterpret_cast<const float4*>(sG + (i + 1) * DV_G + ch);
      const float4 k0 = dv_bf4(sK + i * DC_QS + ch), k1 = dv_bf4(sK + (i + 1) * DC_QS + ch);
      const float4 q0 = dv_bf4(sQ + i * DC_QS + ch), q1 = dv_bf4(sQ + (i + 1) * DC_QS + ch);
      const float4 t = make_float4(exp2f(g1.x - g0.x) * k0.x, exp2f(g1.y - g0.y) * k0.y, exp2f(g1.z - g0.z) * k0.z, exp2f(g1.w - g0.w) * k0.w);
      q00 += q0.x * k0.x + q0.y * k0.y + q0.z * k0.z + q0.w * k0.w;
      q11 += q1.x * k1.x + q1.y * k1.y + q1.z * k1.z + q1.w * k1.w;
      q10 += q1.x * t.x + q1.y * t.y + q1.z * t.z + q1.w * t.w;
      k10 += k1.x * t.x + k1.y * t.y + k1.z * t.z + k1.w * t.w;
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      q00 += __shfl_xor_sync(0xffffffffu, q00, o);
      q11 += __shfl_xor_sync(0xffffffffu, q11, o);
      q10 += __shfl_xor_sync(0xffffffffu, q10, o);
      k10 += __shfl_xor_sync(0xffffffffu, k10, o);
    }
    if ((tid & 7) == 0) {
      Aout[i * DC_C + i] = q00 * (sRq[i] * sRk[i]);
      Aout[(i + 1) * DC_C + i + 1] = q11 * (sRq[i + 1] * sRk[i + 1]);
      Aout[(i + 1) * DC_C + i] = q10 * (sRq[i + 1] * sRk[i]);
      sL[(i + 1) * DP_LT + i] = k10 * (sB[i + 1] * sRk[i + 1] * sRk[i]);
    }
  }
  __syncthreads();
  dc_load_rows<256>(sQ, p.v + row0 * p.v_t + h * p.v_h, p.v_t, n);
  // k_out = k^ e^(G_last - G), and G -> beta k^ e^G in place
#pragma unroll
  for (int e = tid; e < DC_C * 16; e += 256) {
    const int i = e >> 4, j = (e & 15) * 8;
    const float rk = sRk[i], rb = rk * sB[i];
    uint4 u = *reinterpret_cast<const uint4*>(sK + i * DC_QS + j);
    uint32_t* w = reinterpret_cast<uint32_t*>(&u);
    float* gp = sG + i * DV_G + j;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float2 v = unpack_bf16(w[x]);
      const float g0 = gp[2 * x], g1 = gp[2 * x + 1];
      w[x] = pack_bf16(v.x * rk * exp2f(sGL[j + 2 * x] - g0), v.y * rk * exp2f(sGL[j + 2 * x + 1] - g1));
      gp[2 * x] = v.x * rb * exp2f(g0);
      gp[2 * x + 1] = v.y * rb * exp2f(g1);
    }
    *reinterpret_cast<uint4*>(Ko + (hc * DC_C + i) * DC_D + j) = u;
  }
  dc_wait();                                     // v; published by the barriers of the inversion
  dc_invert(sL, sT);
  {
    float* Tout = Tg + hc * DC_C * DC_C;
#pragma unroll
    for (int e = tid; e < DC_C * 16; e += 256) {
      const int i = e >> 4, j = (e & 15) * 4;
      *reinterpret_cast<float4*>(Tout + i * DC_C + j) = *reinterpret_cast<const float4*>(sT + i * DP_LT + j);
    }
  }
  // ---- u = (T beta) v and w = T (beta k^ e^G)
  const int mi = warp < 4 ? warp : 7 - warp, m0 = mi * 16, g = lane >> 2, t2 = (lane & 3) * 2, n0 = (warp >> 2) * 64;
  {
    float acc[8][4] = {};
    for (int kk = 0; kk <= mi; ++kk) {
      uint32_t a[3][4];
      dc_af<3>(a, sT, DP_LT, m0, kk * 16, lane, sB);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t b[4];
        dc_b_t(b, sQ, n0 + np * 16, kk * 16, lane);
        dc_mma31(acc[2 * np], a, b[0], b[1]);
        dc_mma31(acc[2 * np + 1], a, b[2], b[3]);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr)
        *reinterpret_cast<float2*>(U + (hc * DC_C + m0 + g + rr * 8) * DC_D + n0 + nt * 8 + t2) = make_float2(acc[nt][2 * rr], acc[nt][2 * rr + 1]);
  }
  {
    float acc[8][4] = {};
    for (int kk = 0; kk <= mi; ++kk) {
      uint32_t a[3][4];
      dc_af<3>(a, sT, DP_LT, m0, kk * 16, lane);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        uint32_t b[3][2];
        dc_bf_t<3>(b, sG, DV_G, n0 + nt * 8, kk * 16, lane);
        dc_mma33(acc[nt], a, b);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr)
        *reinterpret_cast<uint32_t*>(W + (hc * DC_C + m0 + g + rr * 8) * DC_D + n0 + nt * 8 + t2) = pack_bf16(acc[nt][2 * rr], acc[nt][2 * rr + 1]);
  }
}

// ------------------------------------------------------------------------------------------------
// out: o = (q^ e^G) S + A x, 64 of the 128 value columns per CTA
// ------------------------------------------------------------------------------------------------
// q^ e^G of a chunk into an fp32 tile (over G, which it replaces).  Ends with a barrier.
template <int NT>
__device__ __forceinline__ void dv_q_in(const DeltaChunkIn& p, float* sQi, int ld, float* sRq, int row0, int n, int h) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const __nv_bfloat16* q = p.q + row0 * p.q_t + h * p.q_h;
  dv_cumsum<NT>(p, sQi, ld, row0, n, h);
  for (int r = warp; r < DC_C; r += NT / 32) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < n) v = dv_bf4(q + r * p.q_t + lane * 4);
    const float ss = warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
    const float f = p.l2 ? rsqrtf(ss + 1e-6f) * p.scale : p.scale;
    if (lane == 0) sRq[r] = f;
    float4* at = reinterpret_cast<float4*>(sQi + r * ld + lane * 4);
    const float4 e = *at;
    *at = make_float4(v.x * f * exp2f(e.x), v.y * f * exp2f(e.y), v.z * f * exp2f(e.z), v.w * f * exp2f(e.w));
  }
  __syncthreads();
}

struct VoSmem {
  static constexpr int Q = 0, S = Q + DC_C * DV_A * 4, X = S + DC_D * DO_LD * 4, A = X + DC_C * DO_LD * 4;
  static constexpr int ROWS = A + DC_C * DP_LT * 4;
  static constexpr int TOTAL = ROWS + DC_C * 4;
};

__global__ void __launch_bounds__(256, 2)
delta_vec_out_kernel(const DeltaChunkIn p, const float* __restrict__ Ag, const float* __restrict__ X, const float* __restrict__ St,
                     int nseq, __nv_bfloat16* __restrict__ O) {
  extern __shared__ __align__(16) uint8_t sm[];
  float* sQ = reinterpret_cast<float*>(sm + VoSmem::Q);
  float* sS = reinterpret_cast<float*>(sm + VoSmem::S);
  float* sX = reinterpret_cast<float*>(sm + VoSmem::X);
  float* sA = reinterpret_cast<float*>(sm + VoSmem::A);
  float* sRq = reinterpret_cast<float*>(sm + VoSmem::ROWS);
  const int c = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * 64, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1], slot = c + p.chunk_rows[3 * c + 2];
  const long long hc = static_cast<long long>(h) * p.NC + c;
  dc_load_f32<256, DC_D, 64>(sS, DO_LD, St + ((static_cast<long long>(h) * (p.NC + nseq) + slot) * DC_D) * DC_D + v0, DC_D);
  dc_load_f32<256, DC_C, 64>(sX, DO_LD, X + hc * DC_C * DC_D + v0, DC_D);
  dc_load_f32<256, DC_C, 64>(sA, DP_LT, Ag + hc * DC_C * DC_C, DC_C);
  dv_q_in<256>(p, sQ, DV_A, sRq, row0, n, h);
  const int g = lane >> 2, t2 = (lane & 3) * 2, n0 = warp * 8;
  float acc[4][4] = {};
#pragma unroll 2
  for (int kk = 0; kk < 8; ++kk) {
    uint32_t b[3][2];
    dc_bf_t<3>(b, sS, DO_LD, n0, kk * 16, lane);
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      uint32_t a[3][4];
      dc_af<3>(a, sQ, DV_A, mi * 16, kk * 16, lane);
      dc_mma33(acc[mi], a, b);
    }
  }
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    uint32_t b[3][2];
    dc_bf_t<3>(b, sX, DO_LD, n0, kk * 16, lane);
#pragma unroll
    for (int mi = kk; mi < 4; ++mi) {
      uint32_t a[3][4];
      dc_af<3>(a, sA, DP_LT, mi * 16, kk * 16, lane);
      dc_mma33(acc[mi], a, b);
    }
  }
  __syncthreads();
  __nv_bfloat16* sO = reinterpret_cast<__nv_bfloat16*>(sX);    // [64][72]: whole 128-byte rows go out
#pragma unroll
  for (int mi = 0; mi < 4; ++mi)
#pragma unroll
    for (int rr = 0; rr < 2; ++rr)
      *reinterpret_cast<uint32_t*>(sO + (mi * 16 + g + rr * 8) * 72 + n0 + t2) = pack_bf16(acc[mi][2 * rr], acc[mi][2 * rr + 1]);
  __syncthreads();
#pragma unroll
  for (int e = threadIdx.x; e < DC_C * 8; e += 256) {
    const int i = e >> 3, j = (e & 7) * 8;
    if (i < n)
      *reinterpret_cast<uint4*>(O + (static_cast<long long>(row0 + i) * p.H + h) * DC_D + v0 + j) = *reinterpret_cast<const uint4*>(sO + i * 72 + j);
  }
}

// ------------------------------------------------------------------------------------------------
// bwd_pre: gx = A^T do, gS = (q^ e^G)^T do
// ------------------------------------------------------------------------------------------------
struct VbSmem {
  static constexpr int Q = 0, DO = Q + DC_C * DV_G * 4, A = DO + DC_C * DC_QS * 2, ROWS = A + DC_C * DO_LD * 4;
  static constexpr int TOTAL = ROWS + DC_C * 4;
};

__global__ void __launch_bounds__(256, 2)
delta_vec_bwd_pre_kernel(const DeltaChunkIn p, const __nv_bfloat16* __restrict__ dO, const float* __restrict__ Ag, int nseq,
                         float* __restrict__ GX, float* __restrict__ GS) {
  extern __shared__ __align__(16) uint8_t sm[];
  float* sQ = reinterpret_cast<float*>(sm + VbSmem::Q);
  __nv_bfloat16* sDO = reinterpret_cast<__nv_bfloat16*>(sm + VbSmem::DO);
  float* sA = reinterpret_cast<float*>(sm + VbSmem::A);
  float* sRq = reinterpret_cast<float*>(sm + VbSmem::ROWS);
  const int c = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1], slot = c + p.chunk_rows[3 * c + 2];
  const long long hc = static_cast<long long>(h) * p.NC + c;
  dc_load_rows<256>(sDO, dO + (static_cast<long long>(row0) * p.H + h) * DC_D, static_cast<long long>(p.H) * DC_D, n);
  dc_load_f32<256, DC_C, 64>(sA, DO_LD, Ag + hc * DC_C * DC_C, DC_C);
  dv_q_in<256>(p, sQ, DV_G, sRq, row0, n, h);
  const int g = lane >> 2, t2 = (lane & 3) * 2, n0 = warp * 16;
  uint32_t b[4][4];
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) dc_b_t(b[kk], sDO, n0, kk * 16, lane);
#pragma unroll
  for (int mi = 0; mi < 4; ++mi) {
    float acc[2][4] = {};
#pragma unroll
    for (int kk = mi; kk < 4; ++kk) {
      uint32_t a[3][4];
      dc_af_t<3>(a, sA, DO_LD, mi * 16, kk * 16, lane);
      dc_mma31(acc[0], a, b[kk][0], b[kk][1]);
      dc_mma31(acc[1], a, b[kk][2], b[kk][3]);
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr)
        *reinterpret_cast<float2*>(GX + (hc * DC_C + mi * 16 + g + rr * 8) * DC_D + n0 + nt * 8 + t2) = make_float2(acc[nt][2 * rr], acc[nt][2 * rr + 1]);
  }
  float* out = GS + ((static_cast<long long>(h) * (p.NC + nseq) + slot) * DC_D) * DC_D;
#pragma unroll 2
  for (int mi = 0; mi < 8; ++mi) {
    float acc[2][4] = {};
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t a[3][4];
      dc_af_t<3>(a, sQ, DV_G, mi * 16, kk * 16, lane);
      dc_mma31(acc[0], a, b[kk][0], b[kk][1]);
      dc_mma31(acc[1], a, b[kk][2], b[kk][3]);
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr)
        *reinterpret_cast<float2*>(out + (mi * 16 + g + rr * 8) * DC_D + n0 + nt * 8 + t2) = make_float2(acc[nt][2 * rr], acc[nt][2 * rr + 1]);
  }
}

// ------------------------------------------------------------------------------------------------
// score: db = T^T dx (dv, part of dbeta), dL, dA, and the pairwise sums
//   eq_ic = sum_j dA_ij k^_jc D     eb_ic = sum_j dL_ij k^_jc D     ek_jc = sum_i (dL_ij beta_i k^_ic + dA_ij q^_ic) D
// ------------------------------------------------------------------------------------------------
struct VsSmem {
  static constexpr int Q = 0, K = Q + DC_C * DC_QS * 2, DO = K + DC_C * DC_QS * 2, G = DO + DC_C * DC_QS * 2;
  static constexpr int DX = G + DC_C * DV_G * 4;                      // dx, later the sums ek of the four row groups
  static constexpr int X = DX + DC_C * DV_G * 4, DB = X + DC_C * DV_A * 4;
  static constexpr int PR = DB + DC_C * DV_A * 4;                     // T, then pairs (dL_ij / |k_j|, dA_ij / |k_j|)
  static constexpr int ROWS = PR + 2 * DC_C * DO_LD * 4;
  static constexpr int TOTAL = ROWS + 3 * DC_C * 4 + 4 * DC_C * 4;
};
static_assert(VsSmem::TOTAL <= 232448, "one CTA per SM");

__global__ void __launch_bounds__(512, 1)
delta_vec_score_kernel(const DeltaChunkIn p, const __nv_bfloat16* __restrict__ dO, const float* __restrict__ Tg,
                       const float* __restrict__ X, const float* __restrict__ dX, __nv_bfloat16* __restrict__ dV,
                       float* __restrict__ dBeta, float* __restrict__ DB, float* __restrict__ EQ, float* __restrict__ EB,
                       float* __restrict__ EK) {
  constexpr int NT = 512;
  extern __shared__ __align__(16) uint8_t sm[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(sm + VsSmem::Q);
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(sm + VsSmem::K);
  __nv_bfloat16* sDO = reinterpret_cast<__nv_bfloat16*>(sm + VsSmem::DO);
  float* sG = reinterpret_cast<float*>(sm + VsSmem::G);
  float* sDX = reinterpret_cast<float*>(sm + VsSmem::DX);
  float* sX = reinterpret_cast<float*>(sm + VsSmem::X);
  float* sDB = reinterpret_cast<float*>(sm + VsSmem::DB);
  float* sT = reinterpret_cast<float*>(sm + VsSmem::PR);
  float2* sPR = reinterpret_cast<float2*>(sm + VsSmem::PR);
  float* sB = reinterpret_cast<float*>(sm + VsSmem::ROWS);
  float *sRk = sB + DC_C, *sRq = sRk + DC_C, *sPart = sRq + DC_C;
  const int c = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1];
  const long long hc = static_cast<long long>(h) * p.NC + c;
  dc_load_f32<NT, DC_C, DC_D>(sDX, DV_G, dX + hc * DC_C * DC_D, DC_D);
  dc_load_f32<NT, DC_C, 64>(sT, DO_LD, Tg + hc * DC_C * DC_C, DC_C);
  dc_load_rows<NT>(sQ, p.q + row0 * p.q_t + h * p.q_h, p.q_t, n);
  dc_load_rows<NT>(sK, p.k + row0 * p.k_t + h * p.k_h, p.k_t, n);
  dc_load_rows<NT>(sDO, dO + (static_cast<long long>(row0) * p.H + h) * DC_D, static_cast<long long>(p.H) * DC_D, n);
  dc_load_f32<NT, DC_C, DC_D>(sX, DV_A, X + hc * DC_C * DC_D, DC_D);
  if (tid < DC_C) sB[tid] = tid < n ? __ldg(p.beta + static_cast<long long>(row0 + tid) * p.H + h) : 0.f;
  dv_cumsum<NT>(p, sG, DV_G, row0, n, h);
  dc_row_norms<NT>(sQ, sRq, p.scale, sK, sRk, 1.f, p.l2);
  __syncthreads();
  const int mi = warp >> 2, cq = dc_block_col(warp), m0 = mi * 16, n0 = cq * 32, g = lane >> 2, t2 = (lane & 3) * 2;
  const int i0 = m0 + g, i1 = i0 + 8;
  {
    uint32_t vv[4][2];                           // this thread's v values, on their way during the product
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int i = rr ? i1 : i0;
        vv[nt][rr] = i < n ? __ldg(reinterpret_cast<const uint32_t*>(p.v + (row0 + i) * p.v_t + h * p.v_h + n0 + nt * 8 + t2)) : 0u;
      }
    float acc[4][4] = {}, part[2] = {0.f, 0.f};
    for (int kk = mi; kk < 4; ++kk) {
      uint32_t a[3][4];
      dc_af_t<3>(a, sT, DO_LD, m0, kk * 16, lane);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        uint32_t b[3][2];
        dc_bf_t<3>(b, sDX, DV_G, n0 + nt * 8, kk * 16, lane);
        dc_mma33(acc[nt], a, b);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int col = n0 + nt * 8 + t2;
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int i = rr ? i1 : i0;
        const float x = acc[nt][2 * rr], y = acc[nt][2 * rr + 1], be = sB[i];
        *reinterpret_cast<float2*>(sDB + i * DV_A + col) = make_float2(x, y);
        *reinterpret_cast<float2*>(DB + (hc * DC_C + i) * DC_D + col) = make_float2(x, y);
        if (i < n) {
          const float2 v = unpack_bf16(vv[nt][rr]);
          part[rr] += x * v.x + y * v.y;
          *reinterpret_cast<uint32_t*>(dV + (static_cast<long long>(row0 + i) * p.H + h) * DC_D + col) = pack_bf16(x * be, y * be);
        }
      }
    }
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      float v = part[rr];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if ((lane & 3) == 0) sPart[cq * DC_C + (rr ? i1 : i0)] = v;
    }
  }
  __syncthreads();
  if (tid < n)
    dBeta[static_cast<long long>(row0 + tid) * p.H + h] = (sPart[tid] + sPart[DC_C + tid]) + (sPart[2 * DC_C + tid] + sPart[3 * DC_C + tid]);
  {
    float accP[2][4] = {}, accR[2][4] = {};
    if (cq <= mi) {
#pragma unroll 2
      for (int kk = 0; kk < 8; ++kk) {
        uint32_t ad[4], ab[3][4];
        dc_a(ad, sDO, m0, kk * 16, lane);
        dc_af<3>(ab, sDB, DV_A, m0, kk * 16, lane);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          uint32_t b[3][2];
          dc_bf<3>(b, sX, DV_A, cq * 16 + nt * 8, kk * 16, lane);
          dc_mma13(accR[nt], ad, b);
          dc_mma33(accP[nt], ab, b);
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr)
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int i = rr ? i1 : i0, j = cq * 16 + nt * 8 + t2 + x;
          const float rk = sRk[j];
          sPR[i * DO_LD + j] = make_float2(j < i ? -accP[nt][2 * rr + x] * rk : 0.f, j <= i ? accR[nt][2 * rr + x] * rk : 0.f);
        }
  }
  __syncthreads();
  // ---- pairwise sums: a thread owns one channel and, of every 16 rows, the four of its row group; ek of all 64 rows
  //      accumulates in registers and is added up over the four groups at the end
  const int ch = tid & 127, rg = tid >> 7;
  if (tid < DC_C) sPart[tid] = 1.f / sRk[tid];   // takes |k_j| out of ek again; read behind the barriers of the last loop
  float ek[DC_C];
#pragma unroll
  for (int j = 0; j < DC_C; ++j) ek[j] = 0.f;
#pragma unroll 1
  for (int ib = 0; ib < 4; ++ib) {
    const int ia = ib * 16 + rg * 4;
    float gi[4], kb[4], qh[4], eq[4], eb[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      gi[a] = sG[(ia + a) * DV_G + ch];
      kb[a] = __bfloat162float(sK[(ia + a) * DC_QS + ch]) * (sB[ia + a] * sRk[ia + a]);
      qh[a] = __bfloat162float(sQ[(ia + a) * DC_QS + ch]) * sRq[ia + a];
      eq[a] = eb[a] = 0.f;
    }
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {
      if (jb > ib) continue;
#pragma unroll
      for (int jj = 0; jj < 16; ++jj) {
        const int j = jb * 16 + jj;
        const float gj = sG[j * DV_G + ch], kj = __bfloat162float(sK[j * DC_QS + ch]);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const float2 pr = sPR[(ia + a) * DO_LD + j];       // zero above the diagonal, where the exponent may be positive
          const float e = (jb < ib || j <= ia + a) ? exp2f(gi[a] - gj) : 0.f;
          const float t = e * kj;
          eb[a] = fmaf(pr.x, t, eb[a]);
          eq[a] = fmaf(pr.y, t, eq[a]);
          ek[j] = fmaf(e, fmaf(pr.x, kb[a], pr.y * qh[a]), ek[j]);
        }
      }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      EQ[(hc * DC_C + ia + a) * DC_D + ch] = eq[a];
      EB[(hc * DC_C + ia + a) * DC_D + ch] = eb[a];
    }
  }
#pragma unroll
  for (int grp = 0; grp < 4; ++grp) {
    if (rg == grp) {
#pragma unroll
      for (int j = 0; j < DC_C; ++j) {
        float v = ek[j];
        if (grp > 0) v += sDX[j * DV_G + ch];
        if (grp < 3) sDX[j * DV_G + ch] = v;
        else EK[(hc * DC_C + j) * DC_D + ch] = v * sPart[j];
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------------
// state: products with S and dS, then dq, dk, dg and the rest of dbeta
// ------------------------------------------------------------------------------------------------
struct VtSmem {
  static constexpr int Q = 0, K = Q + DC_C * DC_QS * 2, DO = K + DC_C * DC_QS * 2, G = DO + DC_C * DC_QS * 2;
  static constexpr int X = G + DC_C * DV_G * 4, DB = X + DC_C * DV_A * 4;      // later: gate gradients, out terms
  static constexpr int S = DB + DC_C * DV_A * 4, ROWS = S + DC_D * DV_A * 4;
  static constexpr int DOT = ROWS + 3 * DC_C * 4;
  static constexpr int TOTAL = DOT + DC_D * 4;
  static constexpr int PART = S;                                               // [3][4][64] after the last product
};
static_assert(VtSmem::TOTAL <= 232448, "one CTA per SM");

__global__ void __launch_bounds__(512, 1)
delta_vec_state_kernel(const DeltaChunkIn p, const __nv_bfloat16* __restrict__ dO, const float* __restrict__ X,
                       const float* __restrict__ St, const float* __restrict__ dSt, int nseq, const float* __restrict__ DB,
                       const float* __restrict__ EQ, const float* __restrict__ EB, const float* __restrict__ EK,
                       __nv_bfloat16* __restrict__ dQ, __nv_bfloat16* __restrict__ dK, float* __restrict__ dG, float* __restrict__ dBeta) {
  constexpr int NT = 512;
  extern __shared__ __align__(16) uint8_t sm[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(sm + VtSmem::Q);
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(sm + VtSmem::K);
  __nv_bfloat16* sDO = reinterpret_cast<__nv_bfloat16*>(sm + VtSmem::DO);
  float* sG = reinterpret_cast<float*>(sm + VtSmem::G);
  float* sX = reinterpret_cast<float*>(sm + VtSmem::X);
  float* sDB = reinterpret_cast<float*>(sm + VtSmem::DB);
  float* sS = reinterpret_cast<float*>(sm + VtSmem::S);
  float* sPart = reinterpret_cast<float*>(sm + VtSmem::PART);
  float* sB = reinterpret_cast<float*>(sm + VtSmem::ROWS);
  float *sRk = sB + DC_C, *sRq = sRk + DC_C;
  float* sDot = reinterpret_cast<float*>(sm + VtSmem::DOT);
  const int c = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1], slot = c + p.chunk_rows[3 * c + 2];
  const long long hc = static_cast<long long>(h) * p.NC + c;
  const long long st_at = ((static_cast<long long>(h) * (p.NC + nseq) + slot) * DC_D) * DC_D;
  dc_load_f32<NT, DC_D, DC_D>(sS, DV_A, St + st_at, DC_D);
  dc_load_rows<NT>(sQ, p.q + row0 * p.q_t + h * p.q_h, p.q_t, n);
  dc_load_rows<NT>(sK, p.k + row0 * p.k_t + h * p.k_h, p.k_t, n);
  dc_load_rows<NT>(sDO, dO + (static_cast<long long>(row0) * p.H + h) * DC_D, static_cast<long long>(p.H) * DC_D, n);
  dc_load_f32<NT, DC_C, DC_D>(sX, DV_A, X + hc * DC_C * DC_D, DC_D);
  dc_load_f32<NT, DC_C, DC_D>(sDB, DV_A, DB + hc * DC_C * DC_D, DC_D);
  if (tid < DC_C) sB[tid] = tid < n ? __ldg(p.beta + static_cast<long long>(row0 + tid) * p.H + h) : 0.f;
  dv_cumsum<NT>(p, sG, DV_G, row0, n, h);
  dc_row_norms<NT>(sQ, sRq, p.scale, sK, sRk, 1.f, p.l2);
  __syncthreads();
  const int mi = warp & 3, m0 = mi * 16, cq = warp >> 2, n0 = cq * 32, g = lane >> 2, t2 = (lane & 3) * 2;
  const int i0 = m0 + g, i1 = i0 + 8;
  float part[3][2];
#pragma unroll
  for (int x = 0; x < 3; ++x) part[x][0] = part[x][1] = 0.f;
  float dq[4][4] = {}, dk[4][4] = {};
#pragma unroll 2
  for (int kk = 0; kk < 8; ++kk) {
    uint32_t ad[4], ab[3][4];
    dc_a(ad, sDO, m0, kk * 16, lane);
    dc_af<3>(ab, sDB, DV_A, m0, kk * 16, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      uint32_t b[3][2];
      dc_bf<3>(b, sS, DV_A, n0 + nt * 8, kk * 16, lane);
      dc_mma13(dq[nt], ad, b);
      dc_mma33(dk[nt], ab, b);
    }
  }
  float gate[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int i = rr ? i1 : i0, col = n0 + nt * 8 + t2;
      const long long at = (hc * DC_C + i) * DC_D + col;
      const float2 gg = *reinterpret_cast<const float2*>(sG + i * DV_G + col);
      const float2 eq = __ldg(reinterpret_cast<const float2*>(EQ + at)), eb = __ldg(reinterpret_cast<const float2*>(EB + at));
      const float2 ek = __ldg(reinterpret_cast<const float2*>(EK + at));
      const float2 kf = unpack_bf16(*reinterpret_cast<const uint32_t*>(sK + i * DC_QS + col));
      const float2 qf = unpack_bf16(*reinterpret_cast<const uint32_t*>(sQ + i * DC_QS + col));
      const float be = sB[i], rk = sRk[i], rq = sRq[i];
      const float e0 = exp2f(gg.x), e1 = exp2f(gg.y);
      const float q0 = fmaf(dq[nt][2 * rr], e0, eq.x), q1 = fmaf(dq[nt][2 * rr + 1], e1, eq.y);
      const float b0 = eb.x - dk[nt][2 * rr] * e0, b1 = eb.y - dk[nt][2 * rr + 1] * e1;
      part[0][rr] += qf.x * q0 + qf.y * q1;
      part[1][rr] += kf.x * b0 + kf.y * b1;
      dq[nt][2 * rr] = q0;
      dq[nt][2 * rr + 1] = q1;
      dk[nt][2 * rr] = fmaf(be, b0, ek.x);
      dk[nt][2 * rr + 1] = fmaf(be, b1, ek.y);
      gate[nt][2 * rr] = kf.x * rk * (be * b0 - ek.x) + qf.x * rq * q0;
      gate[nt][2 * rr + 1] = kf.y * rk * (be * b1 - ek.y) + qf.y * rq * q1;
    }
  }
  __syncthreads();                               // S is no longer read by the products
#pragma unroll
  for (int e = 0; e < 8; ++e) {                  // rows of dS replace rows of S; sum_v dS S of every row on the way
    const int r = warp + e * 16;
    float4* at = reinterpret_cast<float4*>(sS + r * DV_A + lane * 4);
    const float4 s = *at, d = __ldg(reinterpret_cast<const float4*>(dSt + st_at + DC_D * DC_D + r * DC_D + lane * 4));
    *at = d;
    const float dot = warp_sum(s.x * d.x + s.y * d.y + s.z * d.z + s.w * d.w);
    if (lane == 0) sDot[r] = dot;
  }
  __syncthreads();
  float out[4][4] = {};
#pragma unroll 2
  for (int kk = 0; kk < 8; ++kk) {
    uint32_t a[3][4];
    dc_af<3>(a, sX, DV_A, m0, kk * 16, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      uint32_t b[3][2];
      dc_bf<3>(b, sS, DV_A, n0 + nt * 8, kk * 16, lane);
      dc_mma33(out[nt], a, b);
    }
  }
  __syncthreads();                               // x, db and dS are no longer read: their space takes the sums below
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int i = rr ? i1 : i0, col = n0 + nt * 8 + t2;
      const float2 gg = *reinterpret_cast<const float2*>(sG + i * DV_G + col), gl = *reinterpret_cast<const float2*>(sG + (DC_C - 1) * DV_G + col);
      const float2 kf = unpack_bf16(*reinterpret_cast<const uint32_t*>(sK + i * DC_QS + col));
      const float x = out[nt][2 * rr] * exp2f(gl.x - gg.x), y = out[nt][2 * rr + 1] * exp2f(gl.y - gg.y);
      const float ox = kf.x * sRk[i] * x, oy = kf.y * sRk[i] * y;
      dk[nt][2 * rr] += x;
      dk[nt][2 * rr + 1] += y;
      part[2][rr] += kf.x * dk[nt][2 * rr] + kf.y * dk[nt][2 * rr + 1];
      *reinterpret_cast<float2*>(sX + i * DV_G + col) = make_float2(gate[nt][2 * rr] - ox, gate[nt][2 * rr + 1] - oy);
      *reinterpret_cast<float2*>(sDB + i * DV_G + col) = make_float2(ox, oy);
    }
  }
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      float v = part[x][rr];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if ((lane & 3) == 0) sPart[(x * 4 + cq) * DC_C + (rr ? i1 : i0)] = v;
    }
  __syncthreads();
  auto row_sum = [&](int x, int i) {
    const float* a = sPart + x * 4 * DC_C + i;
    return (a[0] + a[DC_C]) + (a[2 * DC_C] + a[3 * DC_C]);
  };
#pragma unroll
  for (int rr = 0; rr < 2; ++rr) {
    const int i = rr ? i1 : i0;
    if (i >= n) continue;
    const float rk = sRk[i], rq = sRq[i], r0 = rq / p.scale;
    const float tq = p.l2 ? r0 * r0 * row_sum(0, i) : 0.f, tk = p.l2 ? rk * rk * row_sum(2, i) : 0.f;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int col = n0 + nt * 8 + t2;
      const long long at = (static_cast<long long>(row0 + i) * p.H + h) * DC_D + col;
      const float2 kf = unpack_bf16(*reinterpret_cast<const uint32_t*>(sK + i * DC_QS + col));
      const float2 qf = unpack_bf16(*reinterpret_cast<const uint32_t*>(sQ + i * DC_QS + col));
      *reinterpret_cast<uint32_t*>(dQ + at) = pack_bf16(rq * (dq[nt][2 * rr] - qf.x * tq), rq * (dq[nt][2 * rr + 1] - qf.y * tq));
      *reinterpret_cast<uint32_t*>(dK + at) = pack_bf16(rk * (dk[nt][2 * rr] - kf.x * tk), rk * (dk[nt][2 * rr + 1] - kf.y * tk));
    }
  }
  if (tid < n) dBeta[static_cast<long long>(row0 + tid) * p.H + h] += row_sum(1, tid) * sRk[tid];
  // ---- gates, one channel per thread in each of four row groups: reverse cumulative sums down the rows
  {
    const int ch = tid & 127, rg = tid >> 7;
    float v[16], sum = 0.f, outs = 0.f;
#pragma unroll
    for (int r = 15; r >= 0; --r) {
      sum += sX[(rg * 16 + r) * DV_G + ch];
      v[r] = sum;
      outs += sDB[(rg * 16 + r) * DV_G + ch];
    }
    __syncthreads();
    sX[rg * DV_G + ch] = sum;
    sDB[rg * DV_G + ch] = outs;
    __syncthreads();
    float add = sDot[ch] * exp2f(sG[(DC_C - 1) * DV_G + ch]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      add += sDB[q * DV_G + ch];
      if (q > rg) add += sX[q * DV_G + ch];
    }
    float* dst = dG + (static_cast<long long>(row0) * p.H + h) * DC_D + ch;
#pragma unroll
    for (int r = 0; r < 16; ++r)
      if (rg * 16 + r < n) dst[static_cast<long long>(rg * 16 + r) * p.H * DC_D] = v[r] + add;
  }
}

}  // namespace ttb

using namespace ttb;

// Arguments as in delta_chunk.cu with g fp32 [rows, H, 128] and decay fp32 [H, NC, 128]
TTB_EXPORT int ttb_delta_vec_prep(const DeltaChunkIn* in, float* T, float* A, float* U, void* W, void* Ko, float* decay, void* stream) {
  if (in->rep != 1 || dc_bad(*in)) return 921;
  static bool done[16] = {};
  if (int e = dc_ready(delta_vec_prep_kernel, VpSmem::TOTAL, done)) return e;
  delta_vec_prep_kernel<<<dim3(in->NC, in->H), 256, VpSmem::TOTAL, reinterpret_cast<cudaStream_t>(stream)>>>(
      *in, T, A, U, reinterpret_cast<__nv_bfloat16*>(W), reinterpret_cast<__nv_bfloat16*>(Ko), decay);
  return dc_launched();
}

TTB_EXPORT int ttb_delta_vec_out(const DeltaChunkIn* in, const float* A, const float* X, const float* states, int nseq, void* O, void* stream) {
  if (in->rep != 1 || dc_bad(*in)) return 921;
  static bool done[16] = {};
  if (int e = dc_ready(delta_vec_out_kernel, VoSmem::TOTAL, done)) return e;
  delta_vec_out_kernel<<<dim3(in->NC, in->H, 2), 256, VoSmem::TOTAL, reinterpret_cast<cudaStream_t>(stream)>>>(
      *in, A, X, states, nseq, reinterpret_cast<__nv_bfloat16*>(O));
  return dc_launched();
}

TTB_EXPORT int ttb_delta_vec_bwd_pre(const DeltaChunkIn* in, const void* dO, const float* A, int nseq, float* GX, float* GS, void* stream) {
  if (in->rep != 1 || dc_bad(*in) || (reinterpret_cast<uintptr_t>(dO) & 15)) return 921;
  static bool done[16] = {};
  if (int e = dc_ready(delta_vec_bwd_pre_kernel, VbSmem::TOTAL, done)) return e;
  delta_vec_bwd_pre_kernel<<<dim3(in->NC, in->H), 256, VbSmem::TOTAL, reinterpret_cast<cudaStream_t>(stream)>>>(
      *in, reinterpret_cast<const __nv_bfloat16*>(dO), A, nseq, GX, GS);
  return dc_launched();
}

// scratch: fp32 [4, H, NC, 64, 128]
TTB_EXPORT int ttb_delta_vec_bwd_post(const DeltaChunkIn* in, const void* dO, const float* T, const float* X, const float* dX,
                                      const float* states, const float* dstates, int nseq, void* dQ, void* dK, void* dV, float* dG,
                                      float* dBeta, float* scratch, void* stream) {
  if (in->rep != 1 || dc_bad(*in) || (reinterpret_cast<uintptr_t>(dO) & 15)) return 921;
  static bool done_s[16] = {}, done_t[16] = {};
  if (int e = dc_ready(delta_vec_score_kernel, VsSmem::TOTAL, done_s)) return e;
  if (int e = dc_ready(delta_vec_state_kernel, VtSmem::TOTAL, done_t)) return e;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const dim3 grid(in->NC, in->H);
  const long long n = static_cast<long long>(in->H) * in->NC * DC_C * DC_D;
  float *DB = scratch, *EQ = DB + n, *EB = EQ + n, *EK = EB + n;
  const __nv_bfloat16* d = reinterpret_cast<const __nv_bfloat16*>(dO);
  delta_vec_score_kernel<<<grid, 512, VsSmem::TOTAL, st>>>(*in, d, T, X, dX, reinterpret_cast<__nv_bfloat16*>(dV), dBeta, DB, EQ, EB, EK);
  delta_vec_state_kernel<<<grid, 512, VtSmem::TOTAL, st>>>(*in, d, X, states, dstates, nseq, DB, EQ, EB, EK,
                                                           reinterpret_cast<__nv_bfloat16*>(dQ), reinterpret_cast<__nv_bfloat16*>(dK), dG, dBeta);
  return dc_launched();
}
