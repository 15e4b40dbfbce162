// MoE routing and token permutation kernels for sm_100a.
//
//  * router_fwd / router_bwd: one warp per token does the score function
//    (softmax before or after top-k, or sigmoid), bias-for-selection top-k,
//    probability normalisation, the separate bias-free top-k used by the
//    load-balance loss, per-expert score sums / token counts (padding excluded)
//    and the per-token logsumexp for the z-loss; the backward folds the
//    gradients of the routing weights, of the aux loss and of the z-loss into
//    d(logits).  Semantics: models/modules/moe/router.py:164-380,
//    models/modules/moe/utils.py:127-230, models/modules/moe/moe_utils.py:15-72.
//  * permutation: rows ordered by (expert, token), every expert segment padded
//    to a multiple of 128 rows (pad rows are zero) so that the grouped tcgen05
//    GEMM never straddles experts and the host never learns the split sizes.
//    Contract: ops/moe.py:10-46, ops/providers/native/moe_permutation.py:24-126.
#include "common.cuh"
#include <type_traits>

namespace ttb {

constexpr int MAX_E_PER_LANE = 8;  // E <= 256
constexpr int MAX_K = 16;
constexpr int SEG_ALIGN = 128;

enum ScoreFn : int { SOFTMAX_PRE = 0, SOFTMAX_POST = 1, SIGMOID = 2 };

// Floats as integers in the same order; NaN ranks with -inf (it never wins, but something is always selected), a denormal is zero.
// Zero stands for "none": no float maps to it.
__device__ __forceinline__ unsigned rank_key(float v) {
  unsigned u = __float_as_uint(v == v ? v : -INFINITY);
  if ((u & 0x7fffffffu) < 0x00800000u) u = 0;
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}

// Top-k of `sel` (value j of a lane belongs to expert j * 32 + lane), in descending order, the lower id first among equals: lane r
// returns the r-th id, 0x7fffffff where there is none left.  A round is two warp reductions over integers; as ten shuffles of value and
// id, with the ids in an array that a loop of unknown length indexes, the selection was most of the router's time (below).
template <int EPL>
__device__ __forceinline__ int warp_topk(const float (&sel)[EPL], int E, int k, int lane) {
  unsigned key[EPL];
#pragma unroll
  for (int j = 0; j < EPL; ++j) key[j] = j * 32 + lane < E ? rank_key(sel[j]) : 0u;
  int mine = 0x7fffffff;
  for (int r = 0; r < k; ++r) {
    unsigned best = key[0];
    int bj = 0;
#pragma unroll
    for (int j = 1; j < EPL; ++j)
      if (key[j] > best) { best = key[j]; bj = j; }
    const unsigned top = __reduce_max_sync(0xffffffffu, best);
    const unsigned e = best == top && best != 0u ? bj * 32 + lane : 0x7fffffff;
    const unsigned first = __reduce_min_sync(0xffffffffu, e);
    if (lane == r) mine = static_cast<int>(first);
#pragma unroll
    for (int j = 0; j < EPL; ++j)
      if (first == j * 32 + lane) key[j] = 0u;
  }
  return mine;
}

struct RouterParams {
  const float* logits;      // [T, E] fp32
  const float* expert_bias; // [E] or null (selection only)
  const unsigned char* valid_mask;  // [T] or null (1 = real token) - statistics only
  int* topk_idx;            // [T, k]
  float* topk_prob;         // [T, k]
  float* lse;               // [T] or null
  float* score_partial;     // [grid, E] or null : per-block sum of aux scores (valid tokens)
  int* aux_counts;          // [E] or null : tokens per expert from the bias-free top-k (valid tokens)
  int* counts;              // [E] or null : tokens per expert of the routing top-k (all tokens)
  long long T;
  int E, k, score_fn;
  float scaling;
};

// One warp per token, with the lanes' slots known at compile time (EPL = 1, 2, 4 or 8 for up to 32, 64, 128 or 256 experts).  Bound by the
// chain of the selection's rounds.  4096 tokens, eight of 128 experts: 23 -> 12 us; 16384 tokens, 256 experts, with a bias: 105 -> 54;
// 300 tokens, four of 64: 6.2 -> 3.0.
template <int EPL>
__global__ void __launch_bounds__(256) router_fwd_kernel(const RouterParams p) {
  extern __shared__ float s_scores[];  // [E] block partial
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  if (p.score_partial) {
    for (int i = threadIdx.x; i < p.E; i += blockDim.x) s_scores[i] = 0.f;
    __syncthreads();
  }
  for (long long t = static_cast<long long>(blockIdx.x) * wpb + wib; t < p.T;
       t += static_cast<long long>(gridDim.x) * wpb) {
    float lg[EPL], sc[EPL], sel[EPL];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      int e = j * 32 + lane;
      lg[j] = (e < p.E) ? p.logits[t * p.E + e] : -INFINITY;
      mx = fmaxf(mx, lg[j]);
    }
    mx = warp_max(mx);
    float se = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) se += (lg[j] == -INFINITY) ? 0.f : __expf(lg[j] - mx);
    se = warp_sum(se);
    const float lse = mx + logf(se);
    if (p.lse && lane == 0) p.lse[t] = lse;
    // normalised scores used by the aux loss (and by SOFTMAX_PRE / SIGMOID routing)
    float ssum = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      if (lg[j] == -INFINITY) { sc[j] = 0.f; continue; }
      sc[j] = (p.score_fn == SIGMOID) ? 1.f / (1.f + __expf(-lg[j])) : __expf(lg[j] - lse);
      ssum += sc[j];
    }
    if (p.score_fn == SIGMOID) ssum = warp_sum(ssum);
    // selection values
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      int e = j * 32 + lane;
      float base = (p.score_fn == SOFTMAX_POST) ? lg[j] : sc[j];
      if (lg[j] == -INFINITY) base = -INFINITY;
      else if (p.expert_bias) base += p.expert_bias[e];
      // NaN compares false with everything: the selection below would find no candidate and return an index far
      // outside [0, E).  As -inf a NaN row selects the lowest expert ids; its weights stay NaN and reach the loss.
      sel[j] = (base == base) ? base : -INFINITY;
    }
    const int chosen = warp_topk<EPL>(sel, p.E, p.k, lane);
    // routing weights
    float w = 0.f;  // lane r (< k) holds weight r
    {
      float raw = -INFINITY;
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const float vv = __shfl_sync(0xffffffffu, p.score_fn == SOFTMAX_POST ? lg[j] : sc[j], chosen & 31);
        if (lane < p.k && j == (chosen >> 5)) raw = vv;
      }
      if (p.score_fn == SOFTMAX_POST) {
        float m2 = warp_max(raw);
        float ex = (lane < p.k) ? __expf(raw - m2) : 0.f;
        float s2 = warp_sum(ex);
        w = ex / s2;
      } else if (p.score_fn == SIGMOID) {
        float v2 = (lane < p.k) ? raw : 0.f;
        float s2 = warp_sum(v2);
        w = (p.k > 1) ? v2 / (s2 + 1e-20f) : v2;
      } else {
        w = (lane < p.k) ? raw : 0.f;
      }
      w *= p.scaling;
    }
    const int e_sel = chosen < p.E ? chosen : p.E - 1;   // k > number of selectable experts: stay in range
    if (lane < p.k) {
      p.topk_idx[t * p.k + lane] = e_sel;
      p.topk_prob[t * p.k + lane] = w;
      if (p.counts) atomicAdd(&p.counts[e_sel], 1);
    }
    // aux statistics: bias-free top-k over normalised scores, padding excluded
    const bool valid = p.valid_mask ? (p.valid_mask[t] != 0) : true;
    if ((p.score_partial || p.aux_counts) && valid) {
      float nsc[EPL];
      const float inv = (p.score_fn == SIGMOID) ? 1.f / (ssum + 1e-20f) : 1.f;
#pragma unroll
      for (int j = 0; j < EPL; ++j) nsc[j] = (lg[j] == -INFINITY) ? -INFINITY : sc[j] * inv;
      if (p.aux_counts) {
        const int picked = p.expert_bias ? warp_topk<EPL>(nsc, p.E, p.k, lane) : chosen;
        if (lane < p.k) atomicAdd(&p.aux_counts[picked < p.E ? picked : p.E - 1], 1);
      }
      if (p.score_partial) {
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
          int e = j * 32 + lane;
          if (e < p.E) atomicAdd(&s_scores[e], nsc[j]);
        }
      }
    }
  }
  if (p.score_partial) {
    __syncthreads();
    for (int i = threadIdx.x; i < p.E; i += blockDim.x)
      p.score_partial[static_cast<long long>(blockIdx.x) * p.E + i] = s_scores[i];
  }
}

struct RouterBwdParams {
  const float* logits;     // [T, E]
  const int* topk_idx;     // [T, k]
  const float* topk_prob;  // [T, k] forward output (after scaling)
  const float* dprob;      // [T, k] or null
  const float* aux_grad;   // [E] or null: d(loss)/d(aux score of expert e), applied to valid tokens
  const float* lse;        // unused (kept for ABI symmetry with the forward)
  const unsigned char* valid_mask;
  const float* dlse;       // [T] or null: d(loss)/d(lse_t)
  float* dlogits;          // [T, E] fp32
  long long T;
  int E, k, score_fn;
  float scaling;
};

template <int EPL>
__global__ void __launch_bounds__(256) router_bwd_kernel(const RouterBwdParams p) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (long long t = static_cast<long long>(blockIdx.x) * wpb + (threadIdx.x >> 5); t < p.T;
       t += static_cast<long long>(gridDim.x) * wpb) {
    float lg[EPL], sc[EPL], ds[EPL], dl[EPL];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      int e = j * 32 + lane;
      lg[j] = (e < p.E) ? p.logits[t * p.E + e] : -INFINITY;
      mx = fmaxf(mx, lg[j]);
      ds[j] = 0.f;
      dl[j] = 0.f;
    }
    mx = warp_max(mx);
    float se = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) se += (lg[j] == -INFINITY) ? 0.f : __expf(lg[j] - mx);
    se = warp_sum(se);
    const float lse = mx + logf(se);
    float ssum = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      if (lg[j] == -INFINITY) { sc[j] = 0.f; continue; }
      sc[j] = (p.score_fn == SIGMOID) ? 1.f / (1.f + __expf(-lg[j])) : __expf(lg[j] - lse);
      ssum += sc[j];
    }
    if (p.score_fn == SIGMOID) ssum = warp_sum(ssum);
    const bool valid = p.valid_mask ? (p.valid_mask[t] != 0) : true;

    // ---- routing-weight gradient
    if (p.dprob) {
      // lane r holds (idx_r, w_r, dw_r)
      int my_e = (lane < p.k) ? p.topk_idx[t * p.k + lane] : -1;
      float my_w = (lane < p.k) ? p.topk_prob[t * p.k + lane] / p.scaling : 0.f;  // unscaled weight
      float my_d = (lane < p.k) ? p.dprob[t * p.k + lane] * p.scaling : 0.f;      // grad wrt unscaled weight
      float g_sel = 0.f;  // gradient wrt the selected raw value (logit for POST, score otherwise)
      if (p.score_fn == SOFTMAX_POST) {
        float dot = warp_sum(my_d * my_w);
        g_sel = my_w * (my_d - dot);  // already d(logit)
      } else if (p.score_fn == SIGMOID && p.k > 1) {
        // w_j = s_j / (S + eps): dw/ds_i = (delta_ij - w_j) / (S + eps)
        float S = 0.f;
        {
          float sraw = 0.f;
          for (int r = 0; r < p.k; ++r) {
            int e = __shfl_sync(0xffffffffu, my_e, r);
            float vv = 0.f;
#pragma unroll
            for (int j = 0; j < EPL; ++j)
              if (j == (e >> 5)) vv = sc[j];
            vv = __shfl_sync(0xffffffffu, vv, e & 31);
            if (lane == r) sraw = vv;
          }
          S = warp_sum(sraw) + 1e-20f;
        }
        float dot = warp_sum(my_d * my_w);
        g_sel = (my_d - dot) / S;
      } else {
        g_sel = my_d;
      }
      // scatter g_sel to the owning lane/slot
      for (int r = 0; r < p.k; ++r) {
        int e = __shfl_sync(0xffffffffu, my_e, r);
        float g = __shfl_sync(0xffffffffu, g_sel, r);
        if ((e & 31) == lane) {
#pragma unroll
          for (int j = 0; j < EPL; ++j)
            if (j == (e >> 5)) {
              if (p.score_fn == SOFTMAX_POST) dl[j] += g; else ds[j] += g;
            }
        }
      }
    }
    // ---- aux-loss gradient on normalised scores
    if (p.aux_grad && valid) {
      if (p.score_fn == SIGMOID) {
        // n_e = s_e / (S_all + eps); dn/ds_i = (delta - n_e)/(S_all + eps)
        const float Sall = ssum + 1e-20f;
        float dot = 0.f;
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
          int e = j * 32 + lane;
          if (e < p.E) dot += p.aux_grad[e] * sc[j] / Sall;
        }
        dot = warp_sum(dot);
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
          int e = j * 32 + lane;
          if (e < p.E) ds[j] += (p.aux_grad[e] - dot) / Sall;
        }
      } else {
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
          int e = j * 32 + lane;
          if (e < p.E) ds[j] += p.aux_grad[e];
        }
      }
    }
    // ---- score -> logit jacobian
    if (p.score_fn == SIGMOID) {
#pragma unroll
      for (int j = 0; j < EPL; ++j) dl[j] += ds[j] * sc[j] * (1.f - sc[j]);
    } else {
      float dot = 0.f;
#pragma unroll
      for (int j = 0; j < EPL; ++j) dot += ds[j] * sc[j];
      dot = warp_sum(dot);
#pragma unroll
      for (int j = 0; j < EPL; ++j) dl[j] += sc[j] * (ds[j] - dot);
    }
    // ---- logsumexp gradient (z-loss): d(lse)/dl = softmax(l)
    if (p.dlse) {
      const float zc = p.dlse[t];
#pragma unroll
      for (int j = 0; j < EPL; ++j)
        if (lg[j] != -INFINITY) dl[j] += zc * __expf(lg[j] - lse);
    }
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      int e = j * 32 + lane;
      if (e < p.E) p.dlogits[t * p.E + e] = dl[j];
    }
  }
}

// 32 columns and 32 row groups per block, fixed order (296 x 128 partial sums: 11 us with one thread per column)
__global__ void __launch_bounds__(1024)
colsum_f32_kernel(const float* __restrict__ partial, float* __restrict__ out, int rows, int cols) {
  __shared__ float part[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + x;
  float s = 0.f;
  if (c < cols) {
#pragma unroll 4
    for (int r = y; r < rows; r += 32) s += partial[static_cast<long long>(r) * cols + c];
  }
  part[y][x] = s;
  __syncthreads();
  s = warp_sum(part[x][y]);
  if (x == 0 && blockIdx.x * 32 + y < cols) out[blockIdx.x * 32 + y] = s;
}

// ============================================================================
// Permutation index.  idx: [N] int32 expert ids (N = T*k, token-major).
//   pass 1: counts[e]
//   pass 2: seg_start[E+1] (128-aligned exclusive scan), tile_group[m_tiles_cap],
//           group_rows (== seg_start) and total_rows
//   pass 3: row_of[n] = seg_start[e] + rank of n among entries with expert e (stable)
// ============================================================================
__global__ void perm_count_kernel(const int* __restrict__ idx, long long N, int* __restrict__ counts) {
  __shared__ int red[32];
  const int e = blockIdx.x;
  int c = 0;
#pragma unroll 8
  for (long long i = threadIdx.x; i < N; i += blockDim.x) c += (idx[i] == e);
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x < 32) {
    int v = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) counts[e] = v;
  }
}

__global__ void perm_scan_kernel(const int* __restrict__ counts, int E, int* __restrict__ seg_start,
                                 int* __restrict__ tile_group, int m_tiles_cap, int* __restrict__ status) {
  // single block; E <= 1024
  __shared__ int s_start[1025];
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < E; ++e) {
      s_start[e] = acc;
      acc += ((counts[e] + SEG_ALIGN - 1) / SEG_ALIGN) * SEG_ALIGN;
    }
    s_start[E] = acc;
    if (acc > m_tiles_cap * SEG_ALIGN && status) status[0] = 1;  // capacity exceeded
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= E; i += blockDim.x) seg_start[i] = s_start[i];
  for (int m = threadIdx.x; m < m_tiles_cap; m += blockDim.x) {
    const int row = m * SEG_ALIGN;
    int g = -1;
    if (row < s_start[E]) {
      int lo = 0, hi = E;  // find e with s_start[e] <= row < s_start[e+1]
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (s_start[mid] <= row) lo = mid; else hi = mid;
      }
      g = lo;
    }
    tile_group[m] = g;
  }
}

// Stable ranks: one block of 32 warps per expert, every warp a contiguous span of the entries.  A warp first collects the
// ballots of its span (lane `it` keeps the one of iteration `it`: loads only, no barrier in between), the block adds up the
// spans once, and the second walk hands out rows from the kept ballots.  32768 entries, 128 experts: 66 us with
// 256 threads and two barriers per 256 entries, 7 us now.
constexpr int RANK_THREADS = 1024;

__global__ void __launch_bounds__(RANK_THREADS)
perm_rank_kernel(const int* __restrict__ idx, long long N, const int* __restrict__ seg_start, int* __restrict__ row_of,
                 const int* __restrict__ order_base, int* __restrict__ order) {
  // `order` (optional): the inverse of a second packing of the same entries, order[order_base[e] + rank] = entry
  __shared__ int span[33];          // entries of this expert before every warp's span, then their total
  const int e = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int base = seg_start[e], obase = order ? order_base[e] : 0;
  for (long long s0 = 0; s0 < N;) {
    const long long left = (N - s0 + RANK_THREADS - 1) / RANK_THREADS;
    const int iters = left < 32 ? static_cast<int>(left) : 32;
    const long long w0 = s0 + static_cast<long long>(w) * iters * 32 + lane;
    unsigned mine = 0;
#pragma unroll 8
    for (int it = 0; it < iters; ++it) {
      const long long i = w0 + it * 32;
      const unsigned bal = __ballot_sync(0xffffffffu, i < N && idx[i] == e);
      if (lane == it) mine = bal;
    }
    const int c = __popc(mine);
    int upto = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    if (lane == 31) span[w] = upto;
    __syncthreads();
    if (w == 0) {
      const int v = span[lane];
      int run = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += t;
      }
      span[lane] = run - v;
      if (lane == 31) span[32] = run;
    }
    __syncthreads();
    const int before = span[w];
    for (int it = 0; it < iters; ++it) {
      const unsigned bal = __shfl_sync(0xffffffffu, mine, it);
      if (bal == 0) continue;       // the same on every lane
      const int off = __shfl_sync(0xffffffffu, upto - c, it);
      if ((bal >> lane) & 1u) {
        const int r = before + off + __popc(bal & ((1u << lane) - 1u));
        const long long i = w0 + it * 32;
        row_of[i] = base + r;
        if (order) order[obase + r] = static_cast<int>(i);
      }
    }
    base += span[32];
    obase += span[32];
    s0 += static_cast<long long>(iters) * RANK_THREADS;
    __syncthreads();                // `span` is rewritten by the next round
  }
}

// dst[row_of[n], :] = src[n / k, :]; row_val_out[row_of[n]] = val[n] (optional).  One warp per entry.
__global__ void perm_scatter_kernel(const __nv_bfloat16* __restrict__ src, long long lds,
                                    __nv_bfloat16* __restrict__ dst, long long ldd, const int* __restrict__ row_of,
                                    const float* __restrict__ val, float* __restrict__ row_val_out,
                                    int* __restrict__ row_src_out, long long N, int k, int H) {
  const long long n = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (n >= N) return;
  const long long t = n / k;
  const long long r = row_of[n];
  const uint4* s = reinterpret_cast<const uint4*>(src + t * lds);
  uint4* d = reinterpret_cast<uint4*>(dst + r * ldd);
  for (int c = lane; c < H / 8; c += 32) d[c] = s[c];
  if (lane == 0) {
    if (row_val_out) row_val_out[r] = val[n];
    if (row_src_out) row_src_out[r] = static_cast<int>(n);
  }
}

// zero the pad rows [seg_start[e] + counts[e], seg_start[e+1]) of every expert (their scalars become 0, their return
// tags -1); `zero_ints` (optional, `n_zero` entries) is cleared as well: the progress counters of the next exchange
__global__ void perm_zero_pad_kernel(__nv_bfloat16* __restrict__ dst, long long ldd, const int* __restrict__ counts,
                                     const int* __restrict__ seg_start, float* __restrict__ row_val_out,
                                     int* __restrict__ row_tag_out, int* __restrict__ zero_ints, int n_zero, int H) {
  const int e = blockIdx.x;
  const int r0 = seg_start[e] + counts[e], r1 = seg_start[e + 1];
  const uint4 z = make_uint4(0, 0, 0, 0);
  const int vec = H / 8;
  for (long long i = threadIdx.x; i < static_cast<long long>(r1 - r0) * vec; i += blockDim.x) {
    const long long r = r0 + i / vec;
    reinterpret_cast<uint4*>(dst + r * ldd)[i % vec] = z;
  }
  for (int r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    if (row_val_out) row_val_out[r] = 0.f;
    if (row_tag_out) row_tag_out[r] = -1;
  }
  if (zero_ints)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_zero; i += gridDim.x * blockDim.x) zero_ints[i] = 0;
}

// out[t, :] = sum_j w[t,j] * src[row_of[t*k + j], :] (+ residual[t, :]).  One block per token.
__global__ void perm_combine_kernel(const __nv_bfloat16* __restrict__ src, long long lds,
                                    const int* __restrict__ row_of, const float* __restrict__ w,
                                    const __nv_bfloat16* __restrict__ residual, long long ldr,
                                    __nv_bfloat16* __restrict__ out, long long ldo, int k, int H) {
  const long long t = blockIdx.x;
  for (int c = threadIdx.x * 8; c < H; c += blockDim.x * 8) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int j = 0; j < k; ++j) {
      const long long r = row_of[t * k + j];
      const float wt = w ? w[t * k + j] : 1.f;
      uint4 u = *reinterpret_cast<const uint4*>(src + r * lds + c);
      float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), cc = unpack_bf16(u.z), d = unpack_bf16(u.w);
      acc[0] += wt * a.x; acc[1] += wt * a.y; acc[2] += wt * b.x; acc[3] += wt * b.y;
      acc[4] += wt * cc.x; acc[5] += wt * cc.y; acc[6] += wt * d.x; acc[7] += wt * d.y;
    }
    if (residual) {
      uint4 u = *reinterpret_cast<const uint4*>(residual + t * ldr + c);
      float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), cc = unpack_bf16(u.z), d = unpack_bf16(u.w);
      acc[0] += a.x; acc[1] += a.y; acc[2] += b.x; acc[3] += b.y; acc[4] += cc.x; acc[5] += cc.y; acc[6] += d.x; acc[7] += d.y;
    }
    uint4 o;
    o.x = pack_bf16(acc[0], acc[1]); o.y = pack_bf16(acc[2], acc[3]);
    o.z = pack_bf16(acc[4], acc[5]); o.w = pack_bf16(acc[6], acc[7]);
    *reinterpret_cast<uint4*>(out + t * ldo + c) = o;
  }
}


// ------------------------------------------------------------------------------------------------------------
// Load-balance (auxiliary) loss of one router from the statistics the routing kernel already produced:
//   aux = scale_num * sum_e score_sum[e] * cnt[e] / (k * n^2),   n = max(sum_e cnt[e] / k, 1)
// out[0] = aux, out[1] = aux / coeff (the unscaled value for logging); coef[e] = d aux / d score_sum[e].
// One block.  Replaces a chain of a dozen elementwise / reduction launches per MoE layer
// (models/modules/moe/router.py:164-200 of the reference computes the same quantity with torch ops).
// ------------------------------------------------------------------------------------------------------------
__global__ void aux_loss_kernel(const float* __restrict__ score_sum, const int* __restrict__ cnt, int E, int k,
                                float scale_num, float coeff, float* __restrict__ out, float* __restrict__ coef) {
  __shared__ float red[32];
  __shared__ float s_n, s_dot;
  float c = 0.f, d = 0.f;
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const float ce = static_cast<float>(cnt[e]);
    c += ce;
    d += score_sum[e] * ce;
  }
  c = warp_sum(c);
  d = warp_sum(d);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) red[w] = c;
  __syncthreads();
  if (w == 0) {
    float t = l < nw ? red[l] : 0.f;
    t = warp_sum(t);
    if (l == 0) s_n = fmaxf(t / static_cast<float>(k), 1.f);
  }
  __syncthreads();
  if (l == 0) red[w] = d;
  __syncthreads();
  if (w == 0) {
    float t = l < nw ? red[l] : 0.f;
    t = warp_sum(t);
    if (l == 0) s_dot = t;
  }
  __syncthreads();
  const float f = scale_num / (static_cast<float>(k) * s_n * s_n);
  if (threadIdx.x == 0) {
    out[0] = s_dot * f;
    out[1] = coeff != 0.f ? s_dot * f / coeff : 0.f;
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x) coef[e] = static_cast<float>(cnt[e]) * f;
}

}  // namespace ttb

using namespace ttb;
#define STREAM(s) reinterpret_cast<cudaStream_t>(s)
#define LAUNCH_RET() do { cudaError_t e__ = cudaGetLastError(); return e__ == cudaSuccess ? 0 : 400 + (int)e__; } while (0)

template <typename F>
static void by_slots(int E, F launch) {
  if (E <= 32) launch(std::integral_constant<int, 1>{});
  else if (E <= 64) launch(std::integral_constant<int, 2>{});
  else if (E <= 128) launch(std::integral_constant<int, 4>{});
  else launch(std::integral_constant<int, 8>{});
}

// score_partial: [grid, E] scratch; score_sum: [E] output (may be null together with score_partial)
TTB_EXPORT int ttb_router_fwd(const float* logits, const float* expert_bias, const unsigned char* valid_mask,
                              int* topk_idx, float* topk_prob, float* lse, float* score_partial, float* score_sum,
                              int* aux_counts, int* counts, long long T, int E, int k, int score_fn, float scaling,
                              int grid, void* stream) {
  if (E > 32 * MAX_E_PER_LANE || k > MAX_K || k > E || k > 32) return 901;
  if (T == 0) return 0;
  RouterParams p{logits, expert_bias, valid_mask, topk_idx, topk_prob, lse, score_partial, aux_counts, counts, T, E, k,
                 score_fn, scaling};
  const long long need = (T + 7) / 8;
  if (grid > need) grid = (int)need;
  by_slots(E, [&](auto slots) { router_fwd_kernel<decltype(slots)::value><<<grid, 256, E * sizeof(float), STREAM(stream)>>>(p); });
  if (score_partial && score_sum)
    colsum_f32_kernel<<<(E + 31) / 32, 1024, 0, STREAM(stream)>>>(score_partial, score_sum, grid, E);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_router_bwd(const float* logits, const int* topk_idx, const float* topk_prob, const float* dprob,
                              const float* aux_grad, const float* lse, const unsigned char* valid_mask,
                              const float* dlse, float* dlogits, long long T, int E, int k, int score_fn,
                              float scaling, void* stream) {
  if (E > 32 * MAX_E_PER_LANE || k > MAX_K || k > 32) return 901;
  if (T == 0) return 0;
  RouterBwdParams p{logits, topk_idx, topk_prob, dprob, aux_grad, lse, valid_mask, dlse, dlogits, T, E, k, score_fn,
                    scaling};
  long long grid = (T + 7) / 8;
  if (grid > 4096) grid = 4096;
  by_slots(E, [&](auto slots) { router_bwd_kernel<decltype(slots)::value><<<(unsigned)grid, 256, 0, STREAM(stream)>>>(p); });
  LAUNCH_RET();
}

// Builds the padded (expert, token)-ordered permutation of idx[N].
// counts[E], seg_start[E+1], tile_group[m_tiles_cap], row_of[N], status[1] (set to 1 when capacity is exceeded).
TTB_EXPORT int ttb_perm_index(const int* idx, long long N, int E, int* counts, int* seg_start, int* tile_group,
                              int m_tiles_cap, int* row_of, int* status, void* stream) {
  if (E > 1024) return 901;
  perm_count_kernel<<<E, 1024, 0, STREAM(stream)>>>(idx, N, counts);
  perm_scan_kernel<<<1, 256, 0, STREAM(stream)>>>(counts, E, seg_start, tile_group, m_tiles_cap, status);
  perm_rank_kernel<<<E, RANK_THREADS, 0, STREAM(stream)>>>(idx, N, seg_start, row_of, nullptr, nullptr);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_perm_scatter(const void* src, long long lds, void* dst, long long ldd, const int* row_of,
                                const float* val, float* row_val_out, int* row_src_out, const int* counts,
                                const int* seg_start, int E, long long N, int k, int H, void* stream) {
  if (H % 8 || lds % 8 || ldd % 8) return 901;
  if (counts) perm_zero_pad_kernel<<<E, 1024, 0, STREAM(stream)>>>((__nv_bfloat16*)dst, ldd, counts, seg_start, row_val_out, nullptr, nullptr, 0, H);
  if (N > 0) {
    const long long blocks = (N + 7) / 8;
    perm_scatter_kernel<<<(unsigned)blocks, 256, 0, STREAM(stream)>>>((const __nv_bfloat16*)src, lds,
                                                                     (__nv_bfloat16*)dst, ldd, row_of, val,
                                                                     row_val_out, row_src_out, N, k, H);
  }
  LAUNCH_RET();
}

TTB_EXPORT int ttb_perm_combine(const void* src, long long lds, const int* row_of, const float* w, const void* residual,
                                long long ldr, void* out, long long ldo, long long T, int k, int H, void* stream) {
  if (H % 8 || lds % 8 || ldo % 8) return 901;
  if (T == 0) return 0;
  int threads = H / 8;
  threads = threads > 256 ? 256 : ((threads + 31) / 32) * 32;
  perm_combine_kernel<<<(unsigned)T, threads, 0, STREAM(stream)>>>((const __nv_bfloat16*)src, lds, row_of, w,
                                                                  (const __nv_bfloat16*)residual, ldr,
                                                                  (__nv_bfloat16*)out, ldo, k, H);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_aux_loss(const float* score_sum, const int* cnt, int E, int k, float scale_num, float coeff, float* out2,
                            float* coef, void* stream) {
  if (E < 1 || k < 1) return 901;
  aux_loss_kernel<<<1, 256, 0, STREAM(stream)>>>(score_sum, cnt, E, k, scale_num, coeff, out2, coef);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_moe_seg_align() { return SEG_ALIGN; }

// row_of[n] = base[idx[n]] + stable rank of n among the entries of its expert (base need not be a scan of counts)
TTB_EXPORT int ttb_perm_rank(const int* idx, long long N, int E, const int* base, int* row_of, void* stream) {
  if (N == 0) return 0;
  perm_rank_kernel<<<E, RANK_THREADS, 0, STREAM(stream)>>>(idx, N, base, row_of, nullptr, nullptr);
  LAUNCH_RET();
}

// same, plus order[order_base[idx[n]] + rank] = n : the entries listed in a second (send) order
TTB_EXPORT int ttb_perm_rank_order(const int* idx, long long N, int E, const int* base, int* row_of, const int* order_base,
                                   int* order, void* stream) {
  if (N == 0) return 0;
  perm_rank_kernel<<<E, RANK_THREADS, 0, STREAM(stream)>>>(idx, N, base, row_of, order_base, order);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_perm_zero_pad(void* dst, long long ldd, const int* counts, const int* seg_start, float* row_val,
                                 int E, int H, void* stream) {
  if (H % 8 || ldd % 8) return 901;
  perm_zero_pad_kernel<<<E, 1024, 0, STREAM(stream)>>>((__nv_bfloat16*)dst, ldd, counts, seg_start, row_val, nullptr, nullptr, 0, H);
  LAUNCH_RET();
}

TTB_EXPORT int ttb_perm_zero_pad_tags(void* dst, long long ldd, const int* counts, const int* seg_start, float* row_val,
                                      int* row_tag, int* zero_ints, int n_zero, int E, int H, void* stream) {
  if (H % 8 || ldd % 8) return 901;
  perm_zero_pad_kernel<<<E, 1024, 0, STREAM(stream)>>>((__nv_bfloat16*)dst, ldd, counts, seg_start, row_val, row_tag, zero_ints,
                                                     n_zero, H);
  LAUNCH_RET();
}
