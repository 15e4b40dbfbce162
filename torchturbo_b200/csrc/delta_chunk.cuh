// Chunk-parallel kernels of the gated delta rule for sm_100a: everything around the sequential state recurrence
// (delta_state.cu), one CTA per (64-token chunk, head), forward and backward.  Notation, per chunk and head, with
// rows i, j of the chunk, k^ = k / |k|, q^ = scale q / |q|, G = cumsum(g), D_ij = exp(G_i - G_j), S the state at the
// chunk's start and dS the gradient of the state at its end:
//
//   prep      L_ij = beta_i (k^_i . k^_j) D_ij (i > j)     T = (I + L)^-1      A_ij = (q^_i . k^_j) D_ij (i >= j)
//             u = T (beta v)     w = T (beta k^ e^G)       k_out = k^ e^(G_last - G)
//   out       o = e^G (q^ S) + A x                         (x = u - w S, the "new values", from the recurrence)
//   bwd_pre   gx = A^T do                                  gS = (q^ e^G)^T do
//   bwd_post  db = T^T dx, dL = -strict_lower(db x^T), dA = lower(do x^T), and with them dq, dk, dv, dg, dbeta.
//             (x solves (I + L) x = beta v - (beta k^ e^G) S, so dL needs neither u, w nor another product with T,
//             and d(beta k^ e^G) = -db S^T.)
//
// Arithmetic.  q, k, v and do are bf16 in memory, so they enter the tensor cores exactly; every fp32 operand (T, A,
// S, x and the gradients) is split into three bf16 terms (24 mantissa bits; bwd_post keeps them as planes in shared memory, the
// others split as they load), with three products against an exact operand and six where both sides are fp32.  Norms, decays and masks are applied to fp32 accumulators or fp32 operands,
// never to the bf16 inputs.  Two terms and three products on both-fp32 products left dg 4 to 14 and dbeta 13 to 16 times as
// far from 64 bits as fp32 products; now dbeta, gx and gS are closer than those and dg within 1.5 times of them.
//
// Measured (4096 tokens, 32 heads, four documents, one pass): prep 0.13 ms, out 0.13, bwd_pre 0.09, bwd_post 0.50 (0.15, 0.14, 0.10 and
// 0.58 before the row norms ran beside the loads and the loads that need no row before the rows' own; 0.60 when every warp split
// again the fp32 tiles that it shares with three others).  A gated-delta-net layer forward + backward takes 2.0 ms, against 10.4 when
// the chunk-parallel part was about 250 launches of fp32 products, element-wise passes and gathers over materialised
// [chunk, 64, 64 .. 128] tensors.
//
// Why mma.sync and not tcgen05: the products are 64 x 64 x 128 at most, each feeds the next through registers and shared
// memory, and their operands are built element by element (splits, decays).  What bounds them, from the counters of the same
// case: bwd_post moves 0.69 GB (0.11 ms at the copy rate) and keeps the tensor pipe 34 % active with 12,000 mma.sync per chunk
// and head; one CTA of 16 warps fills 29 % of the issue slots (43 before its planes), and its warps wait for the tensor pipe, for
// results of their own instructions, at barriers between the phases and for loads in similar shares.  out and prep: tensor pipe 30 and 14 %, issue
// slots 49 and 44 %, traffic a third and a quarter of their time.  So neither memory nor the tensor pipe is full: it is the chain
// of phases on one CTA per SM.  That splitting once took only 4 % off bwd_post says the same.
#pragma once
#include "common.cuh"

namespace ttb {

constexpr int DC_C = 64;
constexpr int DC_D = 128;
constexpr int DC_QS = 136;   // row stride (elements) of bf16 tiles: 272 bytes, ldmatrix rows fall on distinct banks

__device__ __forceinline__ void dc_mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t b0, const uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same with a zero accumulator
__device__ __forceinline__ void dc_mul(float (&c)[4], const uint32_t (&a)[4], const uint32_t b0, const uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// Products of operands in bf16 terms, 16 steps of the contraction at a time.  A tensor-core product adds to its accumulator by
// truncation, which over a whole contraction costs more than the roundings of fp32 products do.  So the terms of one step
// start from zero, smallest first, and their sum is added with a rounded fp32 addition.
__device__ __forceinline__ void dc_add(float (&c)[4], const float (&d)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += d[i];
}
// exact x exact
__device__ __forceinline__ void dc_mma11(float (&c)[4], const uint32_t (&a)[4], const uint32_t b0, const uint32_t b1) {
  float d[4];
  dc_mul(d, a, b0, b1);
  dc_add(c, d);
}
// fp32 x exact and exact x fp32 (columns o, o + 1 of the terms): three terms, 24 mantissa bits
__device__ __forceinline__ void dc_mma31(float (&c)[4], const uint32_t (&a)[3][4], const uint32_t b0, const uint32_t b1) {
  float d[4];
  dc_mul(d, a[2], b0, b1);
  dc_mma(d, a[1], b0, b1);
  dc_mma(d, a[0], b0, b1);
  dc_add(c, d);
}
template <int W>
__device__ __forceinline__ void dc_mma13(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[3][W], const int o = 0) {
  float d[4];
  dc_mul(d, a, b[2][o], b[2][o + 1]);
  dc_mma(d, a, b[1][o], b[1][o + 1]);
  dc_mma(d, a, b[0][o], b[0][o + 1]);
  dc_add(c, d);
}
// fp32 x fp32: the six products down to 2^-16 of the leading one; what is left out (mid lo, lo mid, lo lo) lies below the last
// bit of an fp32 product
template <int W>
__device__ __forceinline__ void dc_mma33(float (&c)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][W], const int o = 0) {
  float d[4];
  dc_mul(d, a[2], b[0][o], b[0][o + 1]);
  dc_mma(d, a[1], b[1][o], b[1][o + 1]);
  dc_mma(d, a[0], b[2][o], b[2][o + 1]);
  dc_mma(d, a[1], b[0][o], b[0][o + 1]);
  dc_mma(d, a[0], b[1][o], b[1][o + 1]);
  dc_mma(d, a[0], b[0][o], b[0][o + 1]);
  dc_add(c, d);
}
__device__ __forceinline__ void dc_ldm(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void dc_ldm_t(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
// A fragment (16 rows x 16 k) of a bf16 tile stored [m][k] / of the transpose of one stored [k][m]
__device__ __forceinline__ void dc_a(uint32_t (&r)[4], const __nv_bfloat16* s, int m0, int k0, int lane) {
  dc_ldm(r, s + (m0 + (lane & 15)) * DC_QS + k0 + (lane >> 4) * 8);
}
__device__ __forceinline__ void dc_a_t(uint32_t (&r)[4], const __nv_bfloat16* s, int m0, int k0, int lane) {
  dc_ldm_t(r, s + (k0 + (lane & 7) + ((lane >> 4) << 3)) * DC_QS + m0 + ((lane >> 3) & 1) * 8);
}
// B fragments of two n-tiles (r[0..1], r[2..3]) of a bf16 tile stored [n][k] / stored [k][n]
__device__ __forceinline__ void dc_b(uint32_t (&r)[4], const __nv_bfloat16* s, int n0, int k0, int lane) {
  dc_ldm(r, s + (n0 + (lane & 7) + ((lane >> 4) << 3)) * DC_QS + k0 + ((lane >> 3) & 1) * 8);
}
__device__ __forceinline__ void dc_b_t(uint32_t (&r)[4], const __nv_bfloat16* s, int n0, int k0, int lane) {
  dc_ldm_t(r, s + (k0 + (lane & 15)) * DC_QS + n0 + (lane >> 4) * 8);
}

// (x, y) -> N packed bf16 terms whose sum is (x, y) up to 2^-8N
template <int N>
__device__ __forceinline__ void dc_split(float x, float y, uint32_t (&t)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    t[i] = pack_bf16(x, y);
    if (i + 1 < N) {
      x -= __uint_as_float(t[i] << 16);
      y -= __uint_as_float(t[i] & 0xffff0000u);
    }
  }
}
// A fragment of an fp32 tile, split into N terms.  Stored [m][k]; `cs` (optional) scales column k.
template <int N>
__device__ __forceinline__ void dc_af(uint32_t (&a)[N][4], const float* s, int ld, int m0, int k0, int lane, const float* cs = nullptr) {
  const int g = lane >> 2, t = (lane & 3) * 2;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int k = k0 + t + (r >> 1) * 8;
    float2 v = *reinterpret_cast<const float2*>(s + (m0 + g + (r & 1) * 8) * ld + k);
    if (cs) { v.x *= cs[k]; v.y *= cs[k + 1]; }
    uint32_t w[N];
    dc_split<N>(v.x, v.y, w);
#pragma unroll
    for (int i = 0; i < N; ++i) a[i][r] = w[i];
  }
}
// Same of the transpose of a tile stored [k][m]; `ks` (optional) scales row k.
template <int N>
__device__ __forceinline__ void dc_af_t(uint32_t (&a)[N][4], const float* s, int ld, int m0, int k0, int lane, const float* ks = nullptr) {
  const int g = lane >> 2, t = (lane & 3) * 2;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int k = k0 + t + (r >> 1) * 8, m = m0 + g + (r & 1) * 8;
    float x = s[k * ld + m], y = s[(k + 1) * ld + m];
    if (ks) { x *= ks[k]; y *= ks[k + 1]; }
    uint32_t w[N];
    dc_split<N>(x, y, w);
#pragma unroll
    for (int i = 0; i < N; ++i) a[i][r] = w[i];
  }
}
// B fragment (16 k x 8 n) of an fp32 tile stored [n][k] / stored [k][n], split into N terms
template <int N>
__device__ __forceinline__ void dc_bf(uint32_t (&b)[N][2], const float* s, int ld, int n0, int k0, int lane) {
  const float* p = s + (n0 + (lane >> 2)) * ld + k0 + (lane & 3) * 2;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float2 v = *reinterpret_cast<const float2*>(p + r * 8);
    uint32_t w[N];
    dc_split<N>(v.x, v.y, w);
#pragma unroll
    for (int i = 0; i < N; ++i) b[i][r] = w[i];
  }
}
template <int N>
__device__ __forceinline__ void dc_bf_t(uint32_t (&b)[N][2], const float* s, int ld, int n0, int k0, int lane) {
  const float* p = s + (k0 + (lane & 3) * 2) * ld + n0 + (lane >> 2);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    uint32_t w[N];
    dc_split<N>(p[r * 8 * ld], p[(r * 8 + 1) * ld], w);
#pragma unroll
    for (int i = 0; i < N; ++i) b[i][r] = w[i];
  }
}
// Planes: the three bf16 terms of an fp32 tile, each a bf16 tile of its own (`plane` elements apart, row stride LD), split once
// where the tile is written.  Their fragments come by ldmatrix like those of exact tiles; a fragment of an fp32 tile costs its
// warp about twelve instructions per register, and a tile's fragments are needed by four warps.
__device__ __forceinline__ void dc_put(__nv_bfloat16* s, int plane, float x, float y) {
  uint32_t w[3];
  dc_split<3>(x, y, w);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(s + i * plane) = w[i];
}
__device__ __forceinline__ void dc_put(__nv_bfloat16* s, int plane, float4 v) {
  uint32_t a[3], b[3];
  dc_split<3>(v.x, v.y, a);
  dc_split<3>(v.z, v.w, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(s + i * plane) = make_uint2(a[i], b[i]);
}
// A fragment (16 rows x 16 k) of a tile stored [m][k] / of the transpose of one stored [k][m]
template <int LD>
__device__ __forceinline__ void dc_pa(uint32_t (&r)[3][4], const __nv_bfloat16* s, int plane, int m0, int k0, int lane) {
#pragma unroll
  for (int i = 0; i < 3; ++i) dc_ldm(r[i], s + i * plane + (m0 + (lane & 15)) * LD + k0 + (lane >> 4) * 8);
}
template <int LD>
__device__ __forceinline__ void dc_pa_t(uint32_t (&r)[3][4], const __nv_bfloat16* s, int plane, int m0, int k0, int lane) {
#pragma unroll
  for (int i = 0; i < 3; ++i) dc_ldm_t(r[i], s + i * plane + (k0 + (lane & 7) + ((lane >> 4) << 3)) * LD + m0 + ((lane >> 3) & 1) * 8);
}
// B fragments of two n-tiles (columns 0-1 and 2-3 of r) of a tile stored [n][k] / stored [k][n]
template <int LD>
__device__ __forceinline__ void dc_pb(uint32_t (&r)[3][4], const __nv_bfloat16* s, int plane, int n0, int k0, int lane) {
#pragma unroll
  for (int i = 0; i < 3; ++i) dc_ldm(r[i], s + i * plane + (n0 + (lane & 7) + ((lane >> 4) << 3)) * LD + k0 + ((lane >> 3) & 1) * 8);
}
template <int LD>
__device__ __forceinline__ void dc_pb_t(uint32_t (&r)[3][4], const __nv_bfloat16* s, int plane, int n0, int k0, int lane) {
#pragma unroll
  for (int i = 0; i < 3; ++i) dc_ldm_t(r[i], s + i * plane + (k0 + (lane & 15)) * LD + n0 + (lane >> 4) * 8);
}
// Tiles come in by asynchronous copies, so that all tiles of a kernel are on their way together; `dc_wait` before the barrier
// that publishes them.  64 x 128 bf16 rows of one head -> shared tile; rows past `n` are zero (nothing is read for them).
__device__ __forceinline__ void dc_copy16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void dc_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int NT>
__device__ __forceinline__ void dc_load_rows(__nv_bfloat16* s, const __nv_bfloat16* base, long long row_stride, int n) {
#pragma unroll
  for (int i = threadIdx.x; i < DC_C * 16; i += NT) {
    const int r = i >> 4, c = (i & 15) * 8;
    dc_copy16(s + r * DC_QS + c, base + (r < n ? r * row_stride + c : 0), r < n ? 16 : 0);
  }
}
// fp32 [rows][cols] tile with row stride `src_ld` -> shared with row stride `ld`
template <int NT, int ROWS, int COLS>
__device__ __forceinline__ void dc_load_f32(float* s, int ld, const float* src, int src_ld) {
  constexpr int V = COLS / 4;
#pragma unroll
  for (int i = threadIdx.x; i < ROWS * V; i += NT) {
    const int r = i / V, c = (i - r * V) * 4;
    dc_copy16(s + r * ld + c, src + static_cast<long long>(r) * src_ld + c, 16);
  }
}
// 1 / |row| of a tile (or 1 without normalisation), times `mul`.  All of a warp's rows are summed before the first result is written,
// so that their shuffles overlap; with two tiles in one call those of both.
template <int NT>
__device__ __forceinline__ void dc_row_squares(const __nv_bfloat16* s, float (&ss)[DC_C * 32 / NT]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int x = 0; x < DC_C * 32 / NT; ++x) {
    const uint2 u = *reinterpret_cast<const uint2*>(s + (warp + x * (NT / 32)) * DC_QS + lane * 4);
    const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
    ss[x] = a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y;
  }
}
template <int NT>
__device__ __forceinline__ void dc_row_norms(const __nv_bfloat16* s, float* out, int l2, float mul) {
  float ss[DC_C * 32 / NT];
  dc_row_squares<NT>(s, ss);
#pragma unroll
  for (int x = 0; x < DC_C * 32 / NT; ++x) ss[x] = warp_sum(ss[x]);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int x = 0; x < DC_C * 32 / NT; ++x) out[(threadIdx.x >> 5) + x * (NT / 32)] = l2 ? rsqrtf(ss[x] + 1e-6f) * mul : mul;
  }
}
template <int NT>
__device__ __forceinline__ void dc_row_norms(const __nv_bfloat16* s0, float* out0, float mul0, const __nv_bfloat16* s1, float* out1, float mul1, int l2) {
  float a[DC_C * 32 / NT], b[DC_C * 32 / NT];
  dc_row_squares<NT>(s0, a);
  dc_row_squares<NT>(s1, b);
#pragma unroll
  for (int x = 0; x < DC_C * 32 / NT; ++x) { a[x] = warp_sum(a[x]); b[x] = warp_sum(b[x]); }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int x = 0; x < DC_C * 32 / NT; ++x) {
      const int r = (threadIdx.x >> 5) + x * (NT / 32);
      out0[r] = l2 ? rsqrtf(a[x] + 1e-6f) * mul0 : mul0;
      out1[r] = l2 ? rsqrtf(b[x] + 1e-6f) * mul1 : mul1;
    }
  }
}
// Sixteen warps on 4 x 4 blocks of a 64-row triangle: warp w takes block row w / 4 and this block column.  The work on a triangle grows
// (or falls) with the row, and blocks above the diagonal have none, so the four warps of a scheduler (w % 4) are one of each row, with two
// or three blocks on or below the diagonal.  With the rows dealt out by w % 4 one scheduler had all of the longest.
__device__ __forceinline__ int dc_block_col(int warp) { return (0xE493D2E4u >> ((warp >> 2) * 8 + (warp & 3) * 2)) & 3; }
// inclusive cumulative sum of 64 values, by one warp
__device__ __forceinline__ void dc_cumsum(float* s, int lane) {
  const float a = s[2 * lane], b = s[2 * lane + 1];
  float run = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float up = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += up;
  }
  s[2 * lane] = run - b;
  s[2 * lane + 1] = run;
}
// decay gates and step sizes of the chunk; rows past `n` neither decay nor write (g = beta = 0)
__device__ __forceinline__ void dc_load_gates(const DeltaChunkIn& p, int row0, int n, int h, float* sG, float* sB) {
  if (threadIdx.x < DC_C) {
    const int r = threadIdx.x;
    const long long at = static_cast<long long>(row0 + r) * p.H + h;
    sG[r] = r < n ? __ldg(p.g + at) : 0.f;
    sB[r] = r < n ? __ldg(p.beta + at) : 0.f;
  }
}


constexpr int DP_LT = 72;    // row stride of L, T and A: pairs along a row fall on distinct banks
constexpr int DO_LD = 68;    // row stride of 64-column tiles read down their columns: two rows apart are eight banks apart

// T = (I + L)^-1 of a strictly lower triangular 64 x 64 tile, fp32, by 256 threads: the four 16 x 16 diagonal blocks by
// substitution, then blocks merged 16 -> 32 -> 64, T21 = -T22 (L21 T11); the upper right blocks of L hold the intermediate
// product.  Starts and ends with all threads in step.
__device__ __forceinline__ void dc_invert(float* sL, float* sT) {
  const int tid = threadIdx.x;
  if (tid < 64) {
    const int b0 = (tid >> 4) * 16, col = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s0 = i == col ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
      for (int k = 0; k < i; ++k) {
        const float l = sL[(b0 + i) * DP_LT + b0 + k];
        if (k & 1) s1 = fmaf(-l, x[k], s1); else s0 = fmaf(-l, x[k], s0);
      }
      x[i] = s0 + s1;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) sT[(b0 + i) * DP_LT + b0 + col] = x[i];
  } else {
    for (int e = tid - 64; e < 64 * 64; e += 192) {
      const int i = e >> 6, j = e & 63;
      if ((i >> 4) < (j >> 4)) sT[i * DP_LT + j] = 0.f;
    }
  }
  __syncthreads();
#pragma unroll
  for (int half = 0; half < 2; ++half) {     // half 0: M = L21 T11, half 1: T21 = -T22 M
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int o = tid + e * 256, pr = o >> 8, i = (o >> 4) & 15, j = o & 15, b = pr * 32;
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 16; ++k)
        s = half == 0 ? fmaf(sL[(b + 16 + i) * DP_LT + b + k], sT[(b + k) * DP_LT + b + j], s)
                      : fmaf(-sT[(b + 16 + i) * DP_LT + b + 16 + k], sL[(b + k) * DP_LT + b + 16 + j], s);
      if (half == 0) sL[(b + i) * DP_LT + b + 16 + j] = s; else sT[(b + 16 + i) * DP_LT + b + j] = s;
    }
    __syncthreads();
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int i = tid >> 3, j = (tid & 7) * 4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
      const float l = half == 0 ? sL[(32 + i) * DP_LT + k] : -sT[(32 + i) * DP_LT + 32 + k];
      const float4 r = *reinterpret_cast<const float4*>(half == 0 ? sT + k * DP_LT + j : sL + k * DP_LT + 32 + j);
      s.x = fmaf(l, r.x, s.x); s.y = fmaf(l, r.y, s.y); s.z = fmaf(l, r.z, s.z); s.w = fmaf(l, r.w, s.w);
    }
    *reinterpret_cast<float4*>(half == 0 ? sL + i * DP_LT + 32 + j : sT + (32 + i) * DP_LT + j) = s;
    __syncthreads();
  }
}

template <typename F>
inline int dc_ready(F fn, int bytes, bool (&done)[16]) {
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(fn), bytes, done);
  return e == cudaSuccess ? 0 : 300 + static_cast<int>(e);
}
inline int dc_launched() {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + static_cast<int>(e);
}
inline bool dc_bad(const DeltaChunkIn& a) {
  const uintptr_t p = reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v);
  return (p & 15) || ((a.q_t | a.q_h | a.k_t | a.k_h | a.v_t | a.v_h) & 7) || a.H <= 0 || a.H > 65535 || a.NC <= 0 || a.rep <= 0 || a.H % a.rep;
}

}  // namespace ttb
