// Kernels of the gated delta rule with one decay per head (GatedDeltaNet); the formulas, the arithmetic and the reasons
// are at the top of delta_chunk.cuh.
#include "delta_chunk.cuh"

namespace ttb {

// ------------------------------------------------------------------------------------------------
// prep
// ------------------------------------------------------------------------------------------------
struct DpSmem {
  static constexpr int Q = 0, K = Q + DC_C * DC_QS * 2, V = K + DC_C * DC_QS * 2;
  static constexpr int L = V + DC_C * DC_QS * 2, T = L + DC_C * DP_LT * 4;
  static constexpr int ROWS = T + DC_C * DP_LT * 4;     // G, beta, 1/|k|, 1/|q|, beta e^G / |k|
  static constexpr int TOTAL = ROWS + 5 * DC_C * 4;
};

__global__ void __launch_bounds__(256, 2)
delta_prep_kernel(const DeltaChunkIn p, float* __restrict__ Tg, float* __restrict__ Ag, float* __restrict__ U,
                  __nv_bfloat16* __restrict__ W, __nv_bfloat16* __restrict__ Ko, float* __restrict__ decay) {
  extern __shared__ __align__(16) uint8_t sm[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(sm + DpSmem::Q);
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(sm + DpSmem::K);
  __nv_bfloat16* sV = reinterpret_cast<__nv_bfloat16*>(sm + DpSmem::V);
  float* sL = reinterpret_cast<float*>(sm + DpSmem::L);
  float* sT = reinterpret_cast<float*>(sm + DpSmem::T);
  float* sG = reinterpret_cast<float*>(sm + DpSmem::ROWS);
  float *sB = sG + DC_C, *sRk = sB + DC_C, *sRq = sRk + DC_C, *sW = sRq + DC_C;
  const int c = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1];
  const long long hc = static_cast<long long>(h) * p.NC + c;

  dc_load_rows<256>(sQ, p.q + row0 * p.q_t + h / p.rep * p.q_h, p.q_t, n);
  dc_load_rows<256>(sK, p.k + row0 * p.k_t + h / p.rep * p.k_h, p.k_t, n);
  dc_load_rows<256>(sV, p.v + row0 * p.v_t + h * p.v_h, p.v_t, n);
  dc_load_gates(p, row0, n, h, sG, sB);
  dc_wait();
  __syncthreads();
  dc_row_norms<256>(sQ, sRq, p.scale, sK, sRk, 1.f, p.l2);
  if (warp == 0) dc_cumsum(sG, lane);
  __syncthreads();
  if (tid < DC_C) sW[tid] = sB[tid] * sRk[tid] * expf(sG[tid]);
  if (tid == 0) decay[hc] = expf(sG[DC_C - 1]);

  // rows 16 mi: the work on a triangle grows with mi, so the two warps of a scheduler (warp, warp + 4) take rows that add up
  const int mi = warp < 4 ? warp : 7 - warp, m0 = mi * 16, g = lane >> 2, t2 = (lane & 3) * 2;
  {
    // scores: warps 0-3 k k^T -> L, warps 4-7 q k^T -> A, 16 rows each
    const bool is_q = warp >= 4;
    float acc[8][4] = {};
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      uint32_t a[4];
      dc_a(a, is_q ? sQ : sK, m0, kk * 16, lane);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        if (np > mi) continue;
        uint32_t b[4];
        dc_b(b, sK, np * 16, kk * 16, lane);
        dc_mma11(acc[2 * np], a, b[0], b[1]);
        dc_mma11(acc[2 * np + 1], a, b[2], b[3]);
      }
    }
    float* Aout = Ag + hc * DC_C * DC_C;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int i = m0 + g + rr * 8, j = nt * 8 + t2;
        float2 o = make_float2(0.f, 0.f);
        const float ri = is_q ? sRq[i] : sRk[i] * sB[i];
        if (is_q ? (j <= i) : (j < i)) o.x = acc[nt][2 * rr] * (ri * sRk[j]) * expf(sG[i] - sG[j]);
        if (is_q ? (j + 1 <= i) : (j + 1 < i)) o.y = acc[nt][2 * rr + 1] * (ri * sRk[j + 1]) * expf(sG[i] - sG[j + 1]);
        *reinterpret_cast<float2*>(is_q ? Aout + i * DC_C + j : sL + i * DP_LT + j) = o;
      }
    }
  }
  __syncthreads();
  dc_invert(sL, sT);
  {
    float* Tout = Tg + hc * DC_C * DC_C;
#pragma unroll
    for (int e = tid; e < DC_C * 16; e += 256) {
      const int i = e >> 4, j = (e & 15) * 4;
      *reinterpret_cast<float4*>(Tout + i * DC_C + j) = *reinterpret_cast<const float4*>(sT + i * DP_LT + j);
    }
  }
  // ---- u = (T beta) v, w = (T beta e^G / |k|) k: 16 rows x 64 columns per warp, T lower triangular
  const int n0 = (warp >> 2) * 64;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    float acc[8][4] = {};
    for (int kk = 0; kk <= mi; ++kk) {
      uint32_t a[3][4];
      dc_af<3>(a, sT, DP_LT, m0, kk * 16, lane, which ? sW : sB);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t b[4];
        dc_b_t(b, which ? sK : sV, n0 + np * 16, kk * 16, lane);
        dc_mma31(acc[2 * np], a, b[0], b[1]);
        dc_mma31(acc[2 * np + 1], a, b[2], b[3]);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const long long at = (hc * DC_C + m0 + g + rr * 8) * DC_D + n0 + nt * 8 + t2;
        if (which) *reinterpret_cast<uint32_t*>(W + at) = pack_bf16(acc[nt][2 * rr], acc[nt][2 * rr + 1]);
        else *reinterpret_cast<float2*>(U + at) = make_float2(acc[nt][2 * rr], acc[nt][2 * rr + 1]);
      }
    }
  }
#pragma unroll
  for (int e = tid; e < DC_C * 16; e += 256) {
    const int i = e >> 4, j = (e & 15) * 8;
    const float f = expf(sG[DC_C - 1] - sG[i]) * sRk[i];
    uint4 u = *reinterpret_cast<const uint4*>(sK + i * DC_QS + j);
    uint32_t* w = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float2 v = unpack_bf16(w[x]);
      w[x] = pack_bf16(v.x * f, v.y * f);
    }
    *reinterpret_cast<uint4*>(Ko + (hc * DC_C + i) * DC_D + j) = u;
  }
}

// ------------------------------------------------------------------------------------------------
// out: o = (q e^G / |q|) S + A x, 64 of the 128 value columns per CTA
// ------------------------------------------------------------------------------------------------
struct DoSmem {
  static constexpr int Q = 0, S = Q + DC_C * DC_QS * 2, X = S + DC_D * DO_LD * 4, A = X + DC_C * DO_LD * 4;
  static constexpr int ROWS = A + 3 * DC_C * DP_LT * 2;             // A in planes: all eight warps read all of it
  static constexpr int TOTAL = ROWS + 2 * DC_C * 4;
};

__global__ void __launch_bounds__(256, 2)
delta_out_kernel(const DeltaChunkIn p, const float* __restrict__ Ag, const float* __restrict__ X, const float* __restrict__ St,
                 int nseq, __nv_bfloat16* __restrict__ O) {
  extern __shared__ __align__(16) uint8_t sm[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(sm + DoSmem::Q);
  float* sS = reinterpret_cast<float*>(sm + DoSmem::S);
  float* sX = reinterpret_cast<float*>(sm + DoSmem::X);
  __nv_bfloat16* sA = reinterpret_cast<__nv_bfloat16*>(sm + DoSmem::A);
  float* sG = reinterpret_cast<float*>(sm + DoSmem::ROWS);
  float* sRq = sG + DC_C;
  const int c = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * 64, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1], slot = c + p.chunk_rows[3 * c + 2];
  const long long hc = static_cast<long long>(h) * p.NC + c;
  dc_load_rows<256>(sQ, p.q + row0 * p.q_t + h / p.rep * p.q_h, p.q_t, n);
  dc_load_f32<256, DC_D, 64>(sS, DO_LD, St + ((static_cast<long long>(h) * (p.NC + nseq) + slot) * DC_D) * DC_D + v0, DC_D);
  dc_load_f32<256, DC_C, 64>(sX, DO_LD, X + hc * DC_C * DC_D + v0, DC_D);
  if (threadIdx.x < DC_C) sG[threadIdx.x] = threadIdx.x < n ? __ldg(p.g + static_cast<long long>(row0 + threadIdx.x) * p.H + h) : 0.f;
  {
    float4 va[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) va[e] = __ldg(reinterpret_cast<const float4*>(Ag + hc * DC_C * DC_C) + threadIdx.x + e * 256);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int f = threadIdx.x + e * 256;
      dc_put(sA + (f >> 4) * DP_LT + (f & 15) * 4, DC_C * DP_LT, va[e]);
    }
  }
  dc_wait();
  __syncthreads();
  dc_row_norms<256>(sQ, sRq, p.l2, p.scale);
  if (warp == 0) dc_cumsum(sG, lane);
  __syncthreads();
  const int g = lane >> 2, t2 = (lane & 3) * 2, n0 = warp * 8;
  float acc[4][4] = {};
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    uint32_t b[3][2];
    dc_bf_t<3>(b, sS, DO_LD, n0, kk * 16, lane);
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      uint32_t a[4];
      dc_a(a, sQ, mi * 16, kk * 16, lane);
      dc_mma13(acc[mi], a, b);
    }
  }
#pragma unroll
  for (int mi = 0; mi < 4; ++mi) {
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int i = mi * 16 + g + rr * 8;
      const float f = sRq[i] * expf(sG[i]);
      acc[mi][2 * rr] *= f;
      acc[mi][2 * rr + 1] *= f;
    }
  }
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    uint32_t b[3][2];
    dc_bf_t<3>(b, sX, DO_LD, n0, kk * 16, lane);
#pragma unroll
    for (int mi = kk; mi < 4; ++mi) {
      uint32_t a[3][4];
      dc_pa<DP_LT>(a, sA, DC_C * DP_LT, mi * 16, kk * 16, lane);
      dc_mma33(acc[mi], a, b);
    }
  }
  __syncthreads();
  __nv_bfloat16* sO = sQ;                      // [64][72]: whole 128-byte rows go out
#pragma unroll
  for (int mi = 0; mi < 4; ++mi) {
#pragma unroll
    for (int rr = 0; rr < 2; ++rr)
      *reinterpret_cast<uint32_t*>(sO + (mi * 16 + g + rr * 8) * 72 + n0 + t2) = pack_bf16(acc[mi][2 * rr], acc[mi][2 * rr + 1]);
  }
  __syncthreads();
#pragma unroll
  for (int e = threadIdx.x; e < DC_C * 8; e += 256) {
    const int i = e >> 3, j = (e & 7) * 8;
    if (i < n)
      *reinterpret_cast<uint4*>(O + (static_cast<long long>(row0 + i) * p.H + h) * DC_D + v0 + j) = *reinterpret_cast<const uint4*>(sO + i * 72 + j);
  }
}

// ------------------------------------------------------------------------------------------------
// bwd_pre: gx = A^T do, gS = (q e^G / |q|)^T do, written to the slot of the chunk's start state
// ------------------------------------------------------------------------------------------------
struct DbSmem {
  static constexpr int Q = 0, DO = Q + DC_C * DC_QS * 2, A = DO + DC_C * DC_QS * 2;
  static constexpr int ROWS = A + DC_C * DO_LD * 4;
  static constexpr int TOTAL = ROWS + 3 * DC_C * 4;
};

__global__ void __launch_bounds__(256, 2)
delta_bwd_pre_kernel(const DeltaChunkIn p, const __nv_bfloat16* __restrict__ dO, const float* __restrict__ Ag, int nseq,
                     float* __restrict__ GX, float* __restrict__ GS) {
  extern __shared__ __align__(16) uint8_t sm[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(sm + DbSmem::Q);
  __nv_bfloat16* sDO = reinterpret_cast<__nv_bfloat16*>(sm + DbSmem::DO);
  float* sA = reinterpret_cast<float*>(sm + DbSmem::A);
  float* sG = reinterpret_cast<float*>(sm + DbSmem::ROWS);
  float *sRq = sG + DC_C, *sF = sRq + DC_C;
  const int c = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1], slot = c + p.chunk_rows[3 * c + 2];
  const long long hc = static_cast<long long>(h) * p.NC + c;
  dc_load_rows<256>(sQ, p.q + row0 * p.q_t + h / p.rep * p.q_h, p.q_t, n);
  dc_load_rows<256>(sDO, dO + (static_cast<long long>(row0) * p.H + h) * DC_D, static_cast<long long>(p.H) * DC_D, n);
  dc_load_f32<256, DC_C, 64>(sA, DO_LD, Ag + hc * DC_C * DC_C, DC_C);
  if (threadIdx.x < DC_C) sG[threadIdx.x] = threadIdx.x < n ? __ldg(p.g + static_cast<long long>(row0 + threadIdx.x) * p.H + h) : 0.f;
  dc_wait();
  __syncthreads();
  dc_row_norms<256>(sQ, sRq, p.l2, p.scale);
  if (warp == 0) dc_cumsum(sG, lane);
  __syncthreads();
  if (threadIdx.x < DC_C) sF[threadIdx.x] = sRq[threadIdx.x] * expf(sG[threadIdx.x]);
  __syncthreads();
  const int g = lane >> 2, t2 = (lane & 3) * 2, n0 = warp * 16;
  {
    float acc[4][2][4] = {};
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t b[4];
      dc_b_t(b, sDO, n0, kk * 16, lane);
#pragma unroll
      for (int mi = 0; mi <= kk; ++mi) {           // rows j of A^T meet rows i >= j only
        uint32_t a[3][4];
        dc_af_t<3>(a, sA, DO_LD, mi * 16, kk * 16, lane);
        dc_mma31(acc[mi][0], a, b[0], b[1]);
        dc_mma31(acc[mi][1], a, b[2], b[3]);
      }
    }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int rr = 0; rr < 2; ++rr)
          *reinterpret_cast<float2*>(GX + (hc * DC_C + mi * 16 + g + rr * 8) * DC_D + n0 + nt * 8 + t2) =
              make_float2(acc[mi][nt][2 * rr], acc[mi][nt][2 * rr + 1]);
  }
  {
    // the row factor runs along the contraction, so it rides on do (split in three) and q stays exact
    float acc[8][2][4] = {};
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t b[4], bs[3][4];
      dc_b_t(b, sDO, n0, kk * 16, lane);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int k = kk * 16 + t2 + (r & 1) * 8;
        const float2 v = unpack_bf16(b[r]);
        uint32_t w[3];
        dc_split<3>(v.x * sF[k], v.y * sF[k + 1], w);
#pragma unroll
        for (int i = 0; i < 3; ++i) bs[i][r] = w[i];
      }
#pragma unroll
      for (int mi = 0; mi < 8; ++mi) {
        uint32_t a[4];
        dc_a_t(a, sQ, mi * 16, kk * 16, lane);
        dc_mma13(acc[mi][0], a, bs, 0);
        dc_mma13(acc[mi][1], a, bs, 2);
      }
    }
    float* out = GS + ((static_cast<long long>(h) * (p.NC + nseq) + slot) * DC_D) * DC_D;
#pragma unroll
    for (int mi = 0; mi < 8; ++mi)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int rr = 0; rr < 2; ++rr)
          *reinterpret_cast<float2*>(out + (mi * 16 + g + rr * 8) * DC_D + n0 + nt * 8 + t2) =
              make_float2(acc[mi][nt][2 * rr], acc[mi][nt][2 * rr + 1]);
  }
}

// ------------------------------------------------------------------------------------------------
// bwd_post: dq, dk, dv, dg, dbeta of one chunk and head
// ------------------------------------------------------------------------------------------------
constexpr int DQ_T = 72;                 // row stride of 64-column planes: rows of ldmatrix fall on distinct banks
constexpr int DQ_PT = DC_C * DQ_T;       // elements of one
constexpr int DQ_PL = DC_C * DC_QS;      // elements of a 128-column plane
struct DqSmem {
  static constexpr int Q = 0, K = Q + DQ_PL * 2, DO = K + DQ_PL * 2;
  static constexpr int X = DO + DQ_PL * 2;               // planes of x
  static constexpr int W = X + 3 * DQ_PL * 2;            // planes of dx, then of S and of dS, 64 of the 128 rows at a time (`fetch_half`)
  static constexpr int DB = W + 3 * DQ_PL * 2;           // planes of T, then of db, then of R and P
  static constexpr int ROWS = DB + 6 * DQ_PT * 2;        // G, beta, 1/|k|, scale/|q|, e^G, e^(Gl-G), beta/|k|
  static constexpr int PART = ROWS + 7 * DC_C * 4;       // [6][4][64] row sums per column quarter, [2][64]
  static constexpr int RED = PART + 26 * DC_C * 4;
  static constexpr int TOTAL = RED + 32 * 4;
};
static_assert(2 * DQ_PT >= DQ_PL && DqSmem::TOTAL <= 232448, "one CTA per SM");

__global__ void __launch_bounds__(512, 1)
delta_bwd_post_kernel(const DeltaChunkIn p, const __nv_bfloat16* __restrict__ dO, const float* __restrict__ Tg,
                      const float* __restrict__ X, const float* __restrict__ dX, const float* __restrict__ St,
                      const float* __restrict__ dSt, int nseq, __nv_bfloat16* __restrict__ dQ, __nv_bfloat16* __restrict__ dK,
                      __nv_bfloat16* __restrict__ dV, float* __restrict__ dG, float* __restrict__ dBeta) {
  constexpr int NT = 512;
  extern __shared__ __align__(16) uint8_t sm[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(sm + DqSmem::Q);
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(sm + DqSmem::K);
  __nv_bfloat16* sDO = reinterpret_cast<__nv_bfloat16*>(sm + DqSmem::DO);
  __nv_bfloat16* sX = reinterpret_cast<__nv_bfloat16*>(sm + DqSmem::X);
  __nv_bfloat16* sW = reinterpret_cast<__nv_bfloat16*>(sm + DqSmem::W);
  __nv_bfloat16* sDB = reinterpret_cast<__nv_bfloat16*>(sm + DqSmem::DB);
  __nv_bfloat16 *sR = sDB, *sP = sDB + 3 * DQ_PT;
  float* sPart = reinterpret_cast<float*>(sm + DqSmem::PART);
  float* sG = reinterpret_cast<float*>(sm + DqSmem::ROWS);
  float *sB = sG + DC_C, *sRk = sB + DC_C, *sRq = sRk + DC_C, *sE = sRq + DC_C, *sL = sE + DC_C, *sBk = sL + DC_C;
  float* sRed = reinterpret_cast<float*>(sm + DqSmem::RED);
  const int c = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int row0 = p.chunk_rows[3 * c], n = p.chunk_rows[3 * c + 1], slot = c + p.chunk_rows[3 * c + 2];
  const long long hc = static_cast<long long>(h) * p.NC + c;
  const long long st_at = ((static_cast<long long>(h) * (p.NC + nseq) + slot) * DC_D) * DC_D;
  // 64 rows of 128 columns, four vectors a thread: to registers, and from there to planes
  auto fetch = [&](float4 (&v)[4], const float* src) {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = __ldg(reinterpret_cast<const float4*>(src) + tid + e * NT);
  };
  // 16 of every 32 rows of a 128-row tile, so that each half holds rows of every warp's 32 columns
  auto fetch_half = [&](float4 (&v)[4], const float* src, int half) {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = __ldg(reinterpret_cast<const float4*>(src) + tid + (2 * e + half) * NT);
  };
  auto store = [&](__nv_bfloat16* dst, const float4 (&v)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int f = tid + e * NT;
      dc_put(dst + (f >> 5) * DC_QS + (f & 31) * 4, DQ_PL, v[e]);
    }
  };

  float4 va[4], vb[4];
  {
    // what does not depend on the chunk's rows is asked for first
    float4 vt[2];
    fetch(va, dX + hc * DC_C * DC_D);
    fetch(vb, X + hc * DC_C * DC_D);
#pragma unroll
    for (int e = 0; e < 2; ++e) vt[e] = __ldg(reinterpret_cast<const float4*>(Tg + hc * DC_C * DC_C) + tid + e * NT);
    dc_load_rows<NT>(sQ, p.q + row0 * p.q_t + h / p.rep * p.q_h, p.q_t, n);
    dc_load_rows<NT>(sK, p.k + row0 * p.k_t + h / p.rep * p.k_h, p.k_t, n);
    dc_load_rows<NT>(sDO, dO + (static_cast<long long>(row0) * p.H + h) * DC_D, static_cast<long long>(p.H) * DC_D, n);
    dc_load_gates(p, row0, n, h, sG, sB);
    store(sW, va);
    store(sX, vb);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int f = tid + e * NT;
      dc_put(sDB + (f >> 4) * DQ_T + (f & 15) * 4, DQ_PT, vt[e]);
    }
  }
  fetch_half(va, St + st_at, 0);                 // the first half of S is on its way while db is formed
  dc_wait();
  __syncthreads();
  dc_row_norms<NT>(sQ, sRq, p.scale, sK, sRk, 1.f, p.l2);
  if (warp == 0) dc_cumsum(sG, lane);
  __syncthreads();
  if (tid < DC_C) {
    sE[tid] = expf(sG[tid]);
    sL[tid] = expf(sG[DC_C - 1] - sG[tid]);
    sBk[tid] = sB[tid] * sRk[tid];
  }
  // Warp tile: 16 rows x 32 neighbouring columns, so that a row's sums are four quarters of 32 channels.  (16 columns of each half
  // of the 128 gave the same products but other roundings of those sums: 3e-4 in the 2-norm of a layer's bf16 gradients.)
  const int mi = warp >> 2, cq = dc_block_col(warp);
  const int m0 = mi * 16, n0 = cq * 16, c0 = cq * 32, g = lane >> 2, t2 = (lane & 3) * 2;
  const int i0 = m0 + g, i1 = i0 + 8;
  auto col_of = [&](int nt) { return c0 + nt * 8 + t2; };
  // sums over a row's 128 channels: four lanes, then four warps (added in a fixed order at the end)
  float part[6][2];
#pragma unroll
  for (int x = 0; x < 6; ++x) part[x][0] = part[x][1] = 0.f;
  // ---- db = T^T dx; dv = beta db
  {
    uint32_t vv[4][2];                           // this thread's v values, on their way during the product
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int i = rr ? i1 : i0;
        vv[nt][rr] = i < n ? __ldg(reinterpret_cast<const uint32_t*>(p.v + (row0 + i) * p.v_t + h * p.v_h + col_of(nt))) : 0u;
      }
    float acc[4][4] = {};
    for (int kk = mi; kk < 4; ++kk) {
      uint32_t a[3][4];
      dc_pa_t<DQ_T>(a, sDB, DQ_PT, m0, kk * 16, lane);
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        uint32_t b[3][4];
        dc_pb_t<DC_QS>(b, sW, DQ_PL, c0 + np * 16, kk * 16, lane);
        dc_mma33(acc[2 * np], a, b, 0);
        dc_mma33(acc[2 * np + 1], a, b, 2);
      }
    }
    __syncthreads();                             // dx and T are no longer read: S and db take their places
    store(sW, va);
    fetch_half(va, St + st_at, 1);
    const float be0 = sB[i0], be1 = sB[i1];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int col = col_of(nt);
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int i = rr ? i1 : i0;
        const float x = acc[nt][2 * rr], y = acc[nt][2 * rr + 1], be = rr ? be1 : be0;
        dc_put(sDB + i * DC_QS + col, DQ_PL, x, y);
        if (i < n) {
          const float2 v = unpack_bf16(vv[nt][rr]);
          part[0][rr] += x * v.x + y * v.y;
          *reinterpret_cast<uint32_t*>(dV + (static_cast<long long>(row0 + i) * p.H + h) * DC_D + col) = pack_bf16(x * be, y * be);
        }
      }
    }
  }
  __syncthreads();
  // ---- P = dL . D with dL = -strict_lower(db x^T), R = dA . D with dA = lower(do x^T); 16 x 16 per warp, kept in registers
  // until db has made room for their planes
  float accP[2][4] = {}, accR[2][4] = {};
  if (cq <= mi) {
#pragma unroll 2
    for (int kk = 0; kk < 8; ++kk) {
      uint32_t ad[4], ab[3][4], b[3][4];
      dc_a(ad, sDO, m0, kk * 16, lane);
      dc_pa<DC_QS>(ab, sDB, DQ_PL, m0, kk * 16, lane);
      dc_pb<DC_QS>(b, sX, DQ_PL, n0, kk * 16, lane);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        dc_mma13(accR[nt], ad, b, 2 * nt);
        dc_mma33(accP[nt], ab, b, 2 * nt);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int i = x < 2 ? i0 : i1, j = n0 + nt * 8 + t2 + (x & 1);
        const float d = j <= i ? expf(sG[i] - sG[j]) : 0.f;
        accR[nt][x] = j <= i ? accR[nt][x] * d : 0.f;
        accP[nt][x] = j < i ? -accP[nt][x] * d : 0.f;
      }
    }
  }
  // R and P with column (row) factors, as planes: those of the blocks on and below the diagonal, nothing reads the others
  auto put_scores = [&](bool rows) {
    if (cq > mi) return;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int i = rr ? i1 : i0, j = n0 + nt * 8 + t2;
        const float r0 = rows ? sRq[i] : sRk[j], r1 = rows ? sRq[i] : sRk[j + 1];
        const float p0 = rows ? sBk[i] : sRk[j], p1 = rows ? sBk[i] : sRk[j + 1];
        dc_put(sR + i * DQ_T + j, DQ_PT, accR[nt][2 * rr] * r0, accR[nt][2 * rr + 1] * r1);
        dc_put(sP + i * DQ_T + j, DQ_PT, accP[nt][2 * rr] * p0, accP[nt][2 * rr + 1] * p1);
      }
    }
  };
  // ---- d(q^ e^G) = do S^T, d(beta k^ e^G) = -db S^T, then the score terms R k^, P k^ on the same accumulators
  float dq[4][4] = {}, dk[4][4] = {};
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    if (half == 1) {
      __syncthreads();
      store(sW, va);
      __syncthreads();
    }
#pragma unroll 2
    for (int kk = 0; kk < 8; ++kk) {
      uint32_t ad[4], ab[3][4], b[3][4];
      dc_a(ad, sDO, m0, kk * 16, lane);
      dc_pa<DC_QS>(ab, sDB, DQ_PL, m0, kk * 16, lane);
      dc_pb<DC_QS>(b, sW, DQ_PL, n0, kk * 16, lane);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        dc_mma13(dq[2 * half + nt], ad, b, 2 * nt);
        dc_mma33(dk[2 * half + nt], ab, b, 2 * nt);
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float e = sE[x < 2 ? i0 : i1];
      dq[nt][x] *= e;
      dk[nt][x] *= -e;
    }
  }
  __syncthreads();                               // db and S are no longer read
  put_scores(false);
  // the gradient of the chunk's end state, and S once more for <dS, S>, are fetched while the score terms run
  fetch_half(va, dSt + st_at + DC_D * DC_D, 0);
  fetch_half(vb, St + st_at, 0);
  __syncthreads();
  for (int kk = 0; kk <= mi; ++kk) {
    uint32_t ar[3][4], ap[3][4];
    dc_pa<DQ_T>(ar, sR, DQ_PT, m0, kk * 16, lane);
    dc_pa<DQ_T>(ap, sP, DQ_PT, m0, kk * 16, lane);
#pragma unroll
    for (int np = 0; np < 2; ++np) {
      uint32_t b[4];
      dc_b_t(b, sK, c0 + np * 16, kk * 16, lane);
      dc_mma31(dq[2 * np], ar, b[0], b[1]);
      dc_mma31(dq[2 * np + 1], ar, b[2], b[3]);
      dc_mma31(dk[2 * np], ap, b[0], b[1]);
      dc_mma31(dk[2 * np + 1], ap, b[2], b[3]);
    }
  }
  __syncthreads();
  put_scores(true);
  uint32_t kv[4][2];                             // this thread's k values (bf16 pairs)
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int at = (rr ? i1 : i0) * DC_QS + col_of(nt);
      kv[nt][rr] = *reinterpret_cast<const uint32_t*>(sK + at);
      const float2 kf = unpack_bf16(kv[nt][rr]), qf = unpack_bf16(*reinterpret_cast<const uint32_t*>(sQ + at));
      part[1][rr] += qf.x * dq[nt][2 * rr] + qf.y * dq[nt][2 * rr + 1];
      part[2][rr] += kf.x * dk[nt][2 * rr] + kf.y * dk[nt][2 * rr + 1];
      const float be = sB[rr ? i1 : i0];
      dk[nt][2 * rr] *= be;
      dk[nt][2 * rr + 1] *= be;
    }
  }
  float dots[8];                                 // <dS, S> on the way in, added up in the order of the rows
  auto take_ds = [&](int half) {
    store(sW, va);
#pragma unroll
    for (int e = 0; e < 4; ++e) dots[2 * e + half] = vb[e].x * va[e].x + vb[e].y * va[e].y + vb[e].z * va[e].z + vb[e].w * va[e].w;
  };
  take_ds(0);
  __syncthreads();
  // ---- k in the role of the earlier row: P^T (beta k^) + R^T q^
  {
    float acc[4][4] = {};
    for (int kk = mi; kk < 4; ++kk) {
      uint32_t ar[3][4], ap[3][4];
      dc_pa_t<DQ_T>(ar, sR, DQ_PT, m0, kk * 16, lane);
      dc_pa_t<DQ_T>(ap, sP, DQ_PT, m0, kk * 16, lane);
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        uint32_t bk[4], bq[4];
        dc_b_t(bk, sK, c0 + np * 16, kk * 16, lane);
        dc_b_t(bq, sQ, c0 + np * 16, kk * 16, lane);
        dc_mma31(acc[2 * np], ap, bk[0], bk[1]);
        dc_mma31(acc[2 * np + 1], ap, bk[2], bk[3]);
        dc_mma31(acc[2 * np], ar, bq[0], bq[1]);
        dc_mma31(acc[2 * np + 1], ar, bq[2], bq[3]);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const float2 kf = unpack_bf16(kv[nt][rr]);
        part[3][rr] += kf.x * acc[nt][2 * rr] + kf.y * acc[nt][2 * rr + 1];
        dk[nt][2 * rr] += acc[nt][2 * rr];
        dk[nt][2 * rr + 1] += acc[nt][2 * rr + 1];
      }
  }
  // ---- d(k_out) = x dS^T
  {
    float acc[4][4] = {};
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      if (half == 0) {
        fetch_half(va, dSt + st_at + DC_D * DC_D, 1);
        fetch_half(vb, St + st_at, 1);
      } else {
        __syncthreads();
        take_ds(1);
        __syncthreads();
      }
#pragma unroll 2
      for (int kk = 0; kk < 8; ++kk) {
        uint32_t a[3][4], b[3][4];
        dc_pa<DC_QS>(a, sX, DQ_PL, m0, kk * 16, lane);
        dc_pb<DC_QS>(b, sW, DQ_PL, n0, kk * 16, lane);
        dc_mma33(acc[2 * half], a, b, 0);
        dc_mma33(acc[2 * half + 1], a, b, 2);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const float2 kf = unpack_bf16(kv[nt][rr]);
        const float e = sL[rr ? i1 : i0], x = acc[nt][2 * rr] * e, y = acc[nt][2 * rr + 1] * e;
        part[4][rr] += kf.x * x + kf.y * y;
        dk[nt][2 * rr] += x;
        dk[nt][2 * rr + 1] += y;
        part[5][rr] += kf.x * dk[nt][2 * rr] + kf.y * dk[nt][2 * rr + 1];
      }
  }
  float dot = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) dot += dots[e];
  dot = warp_sum(dot);
  if (lane == 0) sRed[warp] = dot;
#pragma unroll
  for (int x = 0; x < 6; ++x)
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
    const float rk = sRk[i], rq = sRq[i], r0 = rq / p.scale;     // 1/|k|, scale/|q|, 1/|q|
    const float tq = p.l2 ? r0 * r0 * row_sum(1, i) : 0.f, tk = p.l2 ? rk * rk * row_sum(5, i) : 0.f;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int col = col_of(nt);
      const long long at = (static_cast<long long>(row0 + i) * p.H + h) * DC_D + col;
      const float2 kf = unpack_bf16(kv[nt][rr]), qf = unpack_bf16(*reinterpret_cast<const uint32_t*>(sQ + i * DC_QS + col));
      *reinterpret_cast<uint32_t*>(dQ + at) = pack_bf16(rq * (dq[nt][2 * rr] - qf.x * tq), rq * (dq[nt][2 * rr + 1] - qf.y * tq));
      *reinterpret_cast<uint32_t*>(dK + at) = pack_bf16(rk * (dk[nt][2 * rr] - kf.x * tk), rk * (dk[nt][2 * rr + 1] - kf.y * tk));
    }
  }
  // ---- gates: dG_i = kb.dkb + q^.dq^ - k^.(score + out terms); the chunk's last G also carries e^(G_last - G) and decay
  if (warp < 2) {
    const int i = tid;
    const float kb = row_sum(2, i) * sRk[i], out = row_sum(4, i) * sRk[i];
    sPart[24 * DC_C + i] = sB[i] * kb + row_sum(1, i) * sRq[i] - row_sum(3, i) * sRk[i] - out;
    sPart[25 * DC_C + i] = out;
    if (i < n) dBeta[static_cast<long long>(row0 + i) * p.H + h] = row_sum(0, i) + kb;
  }
  __syncthreads();
  if (warp == 0) {
    float total = 0.f;
    if (lane < 16) total = sRed[lane];
    total = warp_sum(total) * sE[DC_C - 1];
    total += warp_sum(sPart[25 * DC_C + lane] + sPart[25 * DC_C + 32 + lane]);
    const float a = sPart[24 * DC_C + 2 * lane], b = sPart[24 * DC_C + 2 * lane + 1];
    float run = a + b;                           // sum from this pair to the chunk's end
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float dn = __shfl_down_sync(0xffffffffu, run, o);
      if (lane + o < 32) run += dn;
    }
    if (2 * lane < n) dG[static_cast<long long>(row0 + 2 * lane) * p.H + h] = run + total;
    if (2 * lane + 1 < n) dG[static_cast<long long>(row0 + 2 * lane + 1) * p.H + h] = run - a + total;
  }
}

// dst[r] = sum of src[r * rep .. r * rep + rep - 1] over rows of 128 channels, for two tensors: the gradients of key heads that
// serve `rep` value heads.  Bound by memory: 16 bytes a thread, summed in fp32 in head order.  4096 rows, 16 key heads of 128 for 32
// value heads: 20 us, where copies of the key heads for every value head took 78 us and the sums over the copies' gradients 70.
__global__ void __launch_bounds__(256)
delta_head_sum_kernel(const __nv_bfloat16* __restrict__ src0, const __nv_bfloat16* __restrict__ src1, __nv_bfloat16* __restrict__ dst0,
                      __nv_bfloat16* __restrict__ dst1, long long vecs, int rep) {
  const __nv_bfloat16* src = blockIdx.y ? src1 : src0;
  __nv_bfloat16* dst = blockIdx.y ? dst1 : dst0;
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= vecs) return;
  const uint4* at = reinterpret_cast<const uint4*>(src) + (i >> 4) * rep * 16 + (i & 15);
  float s[8] = {};
#pragma unroll 4
  for (int x = 0; x < rep; ++x) {
    const uint4 u = at[x * 16];
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 v = unpack_bf16(w[j]);
      s[2 * j] += v.x;
      s[2 * j + 1] += v.y;
    }
  }
  reinterpret_cast<uint4*>(dst)[i] = make_uint4(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]), pack_bf16(s[4], s[5]), pack_bf16(s[6], s[7]));
}

}  // namespace ttb

using namespace ttb;

// src0, src1: bf16 [rows, rep, 128]; dst0, dst1: bf16 [rows, 128], all contiguous on 16 bytes
TTB_EXPORT int ttb_delta_head_sum(const void* src0, const void* src1, void* dst0, void* dst1, long long rows, int rep, void* stream) {
  if (rep < 1 || ((reinterpret_cast<uintptr_t>(src0) | reinterpret_cast<uintptr_t>(src1) | reinterpret_cast<uintptr_t>(dst0) |
                   reinterpret_cast<uintptr_t>(dst1)) & 15)) return 921;
  const long long vecs = rows * 16;
  if (vecs == 0) return 0;
  delta_head_sum_kernel<<<dim3(static_cast<unsigned>((vecs + 255) / 256), 2), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(src0), reinterpret_cast<const __nv_bfloat16*>(src1), reinterpret_cast<__nv_bfloat16*>(dst0),
      reinterpret_cast<__nv_bfloat16*>(dst1), vecs, rep);
  return dc_launched();
}

// T, A: fp32 [H, NC, 64, 64]; U: fp32 [H, NC, 64, 128]; W, K_out: bf16 [H, NC, 64, 128]; decay: fp32 [H, NC]
TTB_EXPORT int ttb_delta_prep(const DeltaChunkIn* in, float* T, float* A, float* U, void* W, void* Ko, float* decay, void* stream) {
  if (dc_bad(*in)) return 921;
  static bool done[16] = {};
  if (int e = dc_ready(delta_prep_kernel, DpSmem::TOTAL, done)) return e;
  delta_prep_kernel<<<dim3(in->NC, in->H), 256, DpSmem::TOTAL, reinterpret_cast<cudaStream_t>(stream)>>>(
      *in, T, A, U, reinterpret_cast<__nv_bfloat16*>(W), reinterpret_cast<__nv_bfloat16*>(Ko), decay);
  return dc_launched();
}

// X: fp32 [H, NC, 64, 128]; states: fp32 [H, NC + nseq, 128, 128]; O: bf16 [rows, H, 128]
TTB_EXPORT int ttb_delta_out(const DeltaChunkIn* in, const float* A, const float* X, const float* states, int nseq, void* O, void* stream) {
  if (dc_bad(*in)) return 921;
  static bool done[16] = {};
  if (int e = dc_ready(delta_out_kernel, DoSmem::TOTAL, done)) return e;
  delta_out_kernel<<<dim3(in->NC, in->H, 2), 256, DoSmem::TOTAL, reinterpret_cast<cudaStream_t>(stream)>>>(
      *in, A, X, states, nseq, reinterpret_cast<__nv_bfloat16*>(O));
  return dc_launched();
}

// dO: bf16 [rows, H, 128] contiguous; GX like X; GS like states (only the slots of chunk starts are written)
TTB_EXPORT int ttb_delta_bwd_pre(const DeltaChunkIn* in, const void* dO, const float* A, int nseq, float* GX, float* GS, void* stream) {
  if (dc_bad(*in) || (reinterpret_cast<uintptr_t>(dO) & 15)) return 921;
  static bool done[16] = {};
  if (int e = dc_ready(delta_bwd_pre_kernel, DbSmem::TOTAL, done)) return e;
  delta_bwd_pre_kernel<<<dim3(in->NC, in->H), 256, DbSmem::TOTAL, reinterpret_cast<cudaStream_t>(stream)>>>(
      *in, reinterpret_cast<const __nv_bfloat16*>(dO), A, nseq, GX, GS);
  return dc_launched();
}

// dQ, dK, dV: bf16 [rows, H, 128]; dG, dBeta: fp32 [rows, H]
TTB_EXPORT int ttb_delta_bwd_post(const DeltaChunkIn* in, const void* dO, const float* T, const float* X, const float* dX,
                                  const float* states, const float* dstates, int nseq, void* dQ, void* dK, void* dV, float* dG,
                                  float* dBeta, void* stream) {
  if (dc_bad(*in) || (reinterpret_cast<uintptr_t>(dO) & 15)) return 921;
  static bool done[16] = {};
  if (int e = dc_ready(delta_bwd_post_kernel, DqSmem::TOTAL, done)) return e;
  delta_bwd_post_kernel<<<dim3(in->NC, in->H), 512, DqSmem::TOTAL, reinterpret_cast<cudaStream_t>(stream)>>>(
      *in, reinterpret_cast<const __nv_bfloat16*>(dO), T, X, dX, states, dstates, nseq, reinterpret_cast<__nv_bfloat16*>(dQ),
      reinterpret_cast<__nv_bfloat16*>(dK), reinterpret_cast<__nv_bfloat16*>(dV), dG, dBeta);
  return dc_launched();
}
