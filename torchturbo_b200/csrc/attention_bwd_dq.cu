// Query-gradient pass of the variable-length flash attention backward for sm_100a: dQ without atomics.
//
// One CTA owns one 128-row query tile of one document for one query head and walks the KV blocks that the tile can
// see, as the forward kernel does; per block, all on tcgen05 with M = 128:
//     S  = Q_i K_j^T            [q, kv]   (K-major x K-major)
//     dP = dO_i V_j^T           [q, kv]   (K-major x K-major)
//     P  = exp2(S c - lse_q),   dS = P (dP - Delta_q) scale     (thread = query row; bf16 pairs written to TMEM)
//     dQ += dS K_j              [q, d]    (A from TMEM, K_j MN-major straight from its [kv, d] tile)
// dQ accumulates in TMEM over the whole tile and is written once, so the result does not depend on the order in which
// CTAs finish: this pass is the bit-reproducible alternative to the atomically reduced dQ of `attn_bwd_kernel`, and
// the only dQ path for query / key heads 192 wide (multi-head latent attention), whose dQ^T, dK and dV accumulators
// do not fit tensor memory together.  It recomputes S and dP (7 products per tile pair over both passes instead of 5).
// Warp roles: 0 TMA producer (Q and dO once, K_j in two stages, V_j in two stages or one for 192-wide heads),
// 1 MMA issuer, 2-9 softmax (warps 2-5 take kv columns 0-63 of the block, warps 6-9 columns 64-127).  Every wait is
// bounded; on a timeout the roles drain to the final barrier, TMEM is freed and the status word records kernel / site.
//
// Bound by the softmax warps: one CTA per SM, two exponentials' worth of arithmetic on each pair of columns against three products.
// Blocks without a mask run a loop without one, the exponential may be moved by the compiler, and dQ leaves through the copy engine in
// place of 64-byte pieces of rows: 98.8 -> 89.6 us for 4096 tokens in three documents with 16 heads of 192 / 128, 527 -> 504 us for one
// document of 8192; 128-wide heads 777 -> 755 (8192 tokens, 32 / 8 heads).
//
// Counterpart of flash-attn 2's backward used through the reference attention interface
// (models/modules/attention/interface.py:114-158), which offers a deterministic mode as well.
#include "common.cuh"
#include <type_traits>

namespace ttb {

constexpr unsigned KID_ATTN_DQ = 5;
constexpr int DQ_TILE = 128 * 128 * 2;   // a [128 x 128] bf16 tile

struct AttnDqParams {
  const int* q_tiles;   // [n_tiles, 3]: first query row, document start, document end
  const float* lse;     // [Hq, T]
  const float* delta;   // [Hq, T]
  __nv_bfloat16* dq;    // [T, Hq, D]
  int Hq, Hk;
  int D, Dv;            // width of query / key heads and of value heads
  long long T;
  float scale;
  int causal;
};

template <int DQK>
struct DqSmem {
  static constexpr int QK_BYTES = 128 * DQK * 2;
  static constexpr int VS = DQK == 128 ? 2 : 1;          // V stages
  static constexpr int Q = 0;
  static constexpr int DO = Q + QK_BYTES;
  static constexpr int K0 = DO + DQ_TILE;
  static constexpr int V0 = K0 + 2 * QK_BYTES;
  static constexpr int BARS = V0 + VS * DQ_TILE;
  static constexpr int TOTAL = BARS + 256 + 1024;
};

__device__ __forceinline__ float dq_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// FULL: heads as wide as the tiles (see attn_bwd_kernel)
template <int DQK, bool FULL>
__global__ void __launch_bounds__(320, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   const __grid_constant__ CUtensorMap tmOut, const AttnDqParams p) {
  using Smem = DqSmem<DQK>;
  const int D = FULL ? DQK : p.D, Dv = FULL ? 128 : p.Dv;
  auto load_head = [](void* dst, const CUtensorMap* map, uint64_t* bar, int col, int head, int width, int row) {
    if (FULL) tma_load_2d(dst, map, bar, head * width + col, row);
    else tma_load_3d(dst, map, bar, col, head, row);
  };
  constexpr int QK_BYTES = Smem::QK_BYTES, VS = Smem::VS, NP = DQK / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::BARS);
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;    // [2]
  uint64_t* k_empty = bars + 3;   // [2]
  uint64_t* v_full = bars + 5;    // [2]
  uint64_t* v_empty = bars + 7;   // [2]
  uint64_t* s_full = bars + 9;    // S and dP of a block are in TMEM
  uint64_t* s_empty = bars + 10;  // every softmax warp has its copy
  uint64_t* ds_full = bars + 11;  // dS of a block is in TMEM
  uint64_t* ds_empty = bars + 12; // dS K of a block retired
  uint64_t* dq_done = bars + 13;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.y, h = blockIdx.x;     // heads vary fastest: the longest tiles of all heads start first
  const int hk = h / (p.Hq / p.Hk);
  const int q0 = p.q_tiles[tile * 3 + 0];
  const int ds = p.q_tiles[tile * 3 + 1];
  const int de = p.q_tiles[tile * 3 + 2];
  const int kv_end = p.causal ? min(de, q0 + 128) : de;
  const int nblk = (kv_end - ds + 127) / 128;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
    }
    mbar_init(s_full, 1); mbar_init(s_empty, 8);
    mbar_init(ds_full, 8); mbar_init(ds_empty, 1);
    mbar_init(dq_done, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tm_S = tmem_base;              // 128 columns
  const uint32_t tm_DP = tmem_base + 128;       // 128 columns
  const uint32_t tm_DQ = tmem_base + 256;       // DQK columns
  const uint32_t tm_DS = tmem_base + 256 + DQK; // 64 columns: bf16 pairs, column = kv index / 2

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
      mbar_expect_tx(q_full, QK_BYTES + DQ_TILE);
#pragma unroll
      for (int pn = 0; pn < NP; ++pn) load_head(smem + Smem::Q + pn * 16384, &tmQ, q_full, pn * 64, h, DQK, q0);
      load_head(smem + Smem::DO, &tmDO, q_full, 0, h, 128, q0);
      load_head(smem + Smem::DO + 16384, &tmDO, q_full, 64, h, 128, q0);
      for (int j = 0; j < nblk; ++j) {
        const int st = j & 1, vs = j % VS;
        const int kv0 = ds + j * 128;
        if (!mbar_wait(&k_empty[st], ((j >> 1) & 1) ^ 1, KID_ATTN_DQ, 1)) break;
        mbar_expect_tx(&k_full[st], QK_BYTES);
#pragma unroll
        for (int pn = 0; pn < NP; ++pn)
          load_head(smem + Smem::K0 + st * QK_BYTES + pn * 16384, &tmK, &k_full[st], pn * 64, hk, DQK, kv0);
        if (!mbar_wait(&v_empty[vs], ((j / VS) & 1) ^ 1, KID_ATTN_DQ, 2)) break;
        mbar_expect_tx(&v_full[vs], DQ_TILE);
        load_head(smem + Smem::V0 + vs * DQ_TILE, &tmV, &v_full[vs], 0, hk, 128, kv0);
        load_head(smem + Smem::V0 + vs * DQ_TILE + 16384, &tmV, &v_full[vs], 64, hk, 128, kv0);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (the whole warp, see umma_ss_w)
    {
      constexpr uint32_t id_s = make_idesc_bf16(128, 128, false, false);
      const uint32_t id_dq = make_idesc_bf16(128, (D + 15) / 16 * 16, false, true);
      const uint32_t leader = elect_one() ? 1u : 0u;
      const SmemDesc dQ = make_smem_desc2(smem_u32(smem + Smem::Q), 16, 1024), dDO = make_smem_desc2(smem_u32(smem + Smem::DO), 16, 1024);
      const SmemDesc dK = make_smem_desc2(smem_u32(smem + Smem::K0), 16, 1024), dV = make_smem_desc2(smem_u32(smem + Smem::V0), 16, 1024);
      const SmemDesc dKt = make_smem_desc2(smem_u32(smem + Smem::K0), 16384, 1024);
      bool ok = mbar_wait(q_full, 0, KID_ATTN_DQ, 3);
      auto issue_scores = [&](int j) -> bool {
        const int st = j & 1, vs = j % VS;
        if (!mbar_wait(&k_full[st], (j >> 1) & 1, KID_ATTN_DQ, 4)) return false;
        if (!mbar_wait(&v_full[vs], (j / VS) & 1, KID_ATTN_DQ, 5)) return false;
        if (!mbar_wait(s_empty, (j & 1) ^ 1, KID_ATTN_DQ, 6)) return false;
        tc_fence_after();
        const SmemDesc k = desc_at(dK, st * QK_BYTES), v = desc_at(dV, vs * DQ_TILE);
#pragma unroll
        for (int kk = 0; kk < DQK / 16; ++kk) {
          const uint32_t off = (kk >> 2) * 16384 + (kk & 3) * 32;
          umma_ss_w(kk * 16 < D ? leader : 0u, tm_S, desc_at(dQ, off), desc_at(k, off), id_s, kk != 0);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (kk >> 2) * 16384 + (kk & 3) * 32;
          umma_ss_w(kk * 16 < Dv ? leader : 0u, tm_DP, desc_at(dDO, off), desc_at(v, off), id_s, kk != 0);
        }
        umma_commit_w(leader, s_full);
        umma_commit_w(leader, &v_empty[vs]);
        return true;
      };
      if (ok && nblk > 0) ok = issue_scores(0);
      for (int j = 0; j < nblk && ok; ++j) {
        if (j + 1 < nblk && !issue_scores(j + 1)) { ok = false; break; }
        if (!mbar_wait(ds_full, j & 1, KID_ATTN_DQ, 7)) { ok = false; break; }
        tc_fence_after();
        const SmemDesc k_t = desc_at(dKt, (j & 1) * QK_BYTES);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          // A = dS from TMEM (a k-step of 16 kv columns is 8 packed columns); B = K: MN-major [kv rows][d], a k-step of
          // 16 kv rows = 2048 bytes, d panels 16 KB apart
          umma_ts_w(leader, tm_DQ, tm_DS + kk * 8, desc_at(k_t, kk * 2048), id_dq, (j | kk) != 0);
        }
        umma_commit_w(leader, &k_empty[j & 1]);
        umma_commit_w(leader, ds_empty);
      }
      if (ok) umma_commit_w(leader, dq_done);
    }
  } else {
    // ---------------------------------------------------------------- softmax / dS (thread = query row, 64 kv columns)
    const int lg = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = lg * 32 + lane;
    const int qrow = q0 + row;
    const bool row_ok = qrow < de;
    const float c = p.scale * 1.4426950408889634f;
    const uint32_t lane_off = static_cast<uint32_t>(lg * 32) << 16;
    const long long stat = static_cast<long long>(h) * p.T + qrow;
    const float neg_lse = row_ok ? -p.lse[stat] * 1.4426950408889634f : -INFINITY;
    const float neg_delta = row_ok ? -p.delta[stat] * p.scale : 0.f;
    const uint64_t cc = f2_pack(c, c), nl = f2_pack(neg_lse, neg_lse);
    const uint64_t sc2 = f2_pack(p.scale, p.scale), nd = f2_pack(neg_delta, neg_delta);
    bool ok = true;
    for (int j = 0; j < nblk; ++j) {
      if (!mbar_wait(s_full, j & 1, KID_ATTN_DQ, 8)) { ok = false; break; }
      tc_fence_after();
      const int kv0 = ds + j * 128 + half * 64;
      float s[64], dp[64];
#pragma unroll
      for (int cb = 0; cb < 2; ++cb) {
        uint32_t va[32], vb[32];
        tmem_ld_32x32b_x32(tm_S + half * 64 + cb * 32 + lane_off, va);
        tmem_ld_32x32b_x32(tm_DP + half * 64 + cb * 32 + lane_off, vb);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          s[cb * 32 + i] = __uint_as_float(va[i]);
          dp[cb * 32 + i] = __uint_as_float(vb[i]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_empty);
      const bool need_mask = (kv0 + 64 > de) || (p.causal && kv0 + 63 > q0);
      const int lim = p.causal ? min(de - 1, qrow) : de - 1;  // last visible kv index
      uint32_t w[32];
      // masked blocks have their own copy: a branch around every pair of columns kept their chains from overlapping
      auto columns = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          float a0, a1;
          f2_unpack(f2_fma(f2_pack(s[2 * i], s[2 * i + 1]), cc, nl), a0, a1);
          float p0 = dq_exp2(a0), p1 = dq_exp2(a1);
          if (decltype(masked)::value) {
            p0 = (row_ok && kv0 + 2 * i <= lim) ? p0 : 0.f;
            p1 = (row_ok && kv0 + 2 * i + 1 <= lim) ? p1 : 0.f;
          }
          float d0, d1;
          f2_unpack(f2_mul(f2_pack(p0, p1), f2_fma(f2_pack(dp[2 * i], dp[2 * i + 1]), sc2, nd)), d0, d1);
          w[i] = pack_bf16(d0, d1);
        }
      };
      if (need_mask) columns(std::true_type{});
      else columns(std::false_type{});
      // the dS buffer was read by the product of the previous block
      if (j > 0) {
        if (!mbar_wait(ds_empty, (j - 1) & 1, KID_ATTN_DQ, 9)) { ok = false; break; }
        tc_fence_after();
      }
      tmem_st_32x32b_x32(tm_DS + half * 32 + lane_off, w);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    // ---- epilogue: each half writes its share of the dQ columns, 32 at a time, by way of shared memory (all loads have been used) and
    // the copy engine; rows of a tile that ends in another document, which that document's CTA writes, one by one
    if (ok && nblk > 0) ok = mbar_wait(dq_done, 0, KID_ATTN_DQ, 10);
    if (ok && nblk > 0) {
      tc_fence_after();
      constexpr int COLS = DQK / 2;               // 64 or 96 columns per half
      const bool whole = q0 + lg * 32 + 32 <= de;
      uint8_t* tile = smem + (half * 4 + lg) * (COLS / 32) * 2048;
      __nv_bfloat16* dst = p.dq + (static_cast<long long>(qrow) * p.Hq + h) * D + half * COLS;
#pragma unroll
      for (int cb = 0; cb < COLS / 32; ++cb) {
        const int col = half * COLS + cb * 32;
        if (col >= D) break;                      // uniform
        uint32_t v[32];
        tmem_ld_32x32b_x32(tm_DQ + col + lane_off, v);
        tmem_ld_wait();
        uint8_t* box = tile + cb * 2048;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float* f = reinterpret_cast<const float*>(v + 8 * i);
          const uint4 o = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
          if (whole) st_shared_v4(smem_u32(box) + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4), o.x, o.y, o.z, o.w);
          else if (row_ok && col + 8 * i < D) *reinterpret_cast<uint4*>(dst + cb * 32 + 8 * i) = o;
        }
        if (whole) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (FULL) tma_store_2d(&tmOut, box, h * D + col, q0 + lg * 32);
            else tma_store_3d(&tmOut, box, col, h, q0 + lg * 32);
            bulk_commit_group();
          }
        }
      }
      if (lane == 0) bulk_wait_read_all();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int DQK, bool FULL>
static int launch_attn_dq(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tk, const CUtensorMap& tv,
                          const CUtensorMap& tout, const AttnDqParams& p, int n_tiles, cudaStream_t stream) {
  static bool smem_done[16] = {};
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(attn_bwd_dq_kernel<DQK, FULL>), DqSmem<DQK>::TOTAL, smem_done);
  if (e != cudaSuccess) return 300 + static_cast<int>(e);
  dim3 grid(p.Hq, n_tiles);
  attn_bwd_dq_kernel<DQK, FULL><<<grid, 320, DqSmem<DQK>::TOTAL, stream>>>(tq, tdo, tk, tv, tout, p);
  return 0;
}

}  // namespace ttb

using namespace ttb;

// q: [T, Hq, D] contiguous; dout: [T, Hq, Dv] contiguous; k: [T, Hk, D] (ldk); v: [T, Hk, Dv] (ldv); lse, delta:
// fp32 [Hq, T] (delta = rowsum(dO * O), from the backward's row-dot kernel); dq: bf16 [T, Hq, D], rows outside every
// document are not written.  D and Dv as for ttb_attn_bwd.
TTB_EXPORT int ttb_attn_bwd_dq(const void* q, const void* k, long long ldk, const void* v, long long ldv, const void* dout,
                               const float* lse, const float* delta, void* dq, const int* q_tiles, int n_tiles, long long T,
                               int Hq, int Hk, int D, int Dv, float scale, int causal, void* stream_ptr) {
  if (D < 8 || Dv < 8 || D % 8 || Dv % 8 || Dv > 128 || (D > 128 && !(D == 192 && Dv == 128)) || Hq % Hk) return 901;
  if ((ldk % 8) || (ldv % 8)) return 902;
  if (T == 0 || n_tiles == 0) return 0;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  const bool full = D >= 128 && Dv == 128;
  const auto map = full ? make_rows_map : make_heads_map;
  CUtensorMap tq, tdo, tk, tv;
  if (map(&tq, q, T, (long long)Hq * D, Hq, D, 128)) return 101;
  if (map(&tdo, dout, T, (long long)Hq * Dv, Hq, Dv, 128)) return 102;
  if (map(&tk, k, T, ldk, Hk, D, 128)) return 103;
  if (map(&tv, v, T, ldv, Hk, Dv, 128)) return 104;
  CUtensorMap tout;
  {
    const uint64_t dims2[2] = {static_cast<uint64_t>(Hq) * D, static_cast<uint64_t>(T)};
    const uint64_t dims3[3] = {static_cast<uint64_t>(D), static_cast<uint64_t>(Hq), static_cast<uint64_t>(T)};
    const uint64_t str[2] = {static_cast<uint64_t>(D) * 2, static_cast<uint64_t>(Hq) * D * 2};
    const uint32_t box2[2] = {32, 32}, box3[3] = {32, 1, 32};
    if (make_tmap_typed(&tout, dq, full ? 2 : 3, full ? dims2 : dims3, full ? str + 1 : str, full ? box2 : box3,
                        CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, CU_TENSOR_MAP_SWIZZLE_64B))
      return 105;
  }
  AttnDqParams p{q_tiles, lse, delta, (__nv_bfloat16*)dq, Hq, Hk, D, Dv, T, scale, causal};
  const int rc = D == 192 ? launch_attn_dq<192, true>(tq, tdo, tk, tv, tout, p, n_tiles, stream)
                          : (full ? launch_attn_dq<128, true>(tq, tdo, tk, tv, tout, p, n_tiles, stream)
                                  : launch_attn_dq<128, false>(tq, tdo, tk, tv, tout, p, n_tiles, stream));
  if (rc) return rc;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}
