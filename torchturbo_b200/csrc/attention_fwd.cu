// Variable-length (packed) flash attention forward for sm_100a, GQA, causal or full; heads up to 128 wide (narrow ones, 72 in a
// ViT, in multiples of 8: the tiles' missing columns read as zero and take no part in the products beyond the next multiple of
// 16), or value heads 128 wide with query / key heads 192 (multi-head latent attention: 128 without position + 64 rotary).
// Padding the heads first cost a ViT block (16 heads of 72, 3000 rows, forward + backward) 12 launches and 120 of 1063 us on the
// device; the kernels themselves take the same time.
//
// One CTA handles two neighbouring 128-row query tiles of one document for one query head, or one.  Warp roles:
//   warp 0      TMA producer   : Q once, then K_j / V_j tiles, shared by both query tiles
//   warp 1      MMA issuer     : S = Q_t K_j^T (tcgen05, fp32 in TMEM) and O_t += P V_j (P read from TMEM, V MN-major
//                                straight from its [kv, d] tile; O_t stays in TMEM)
//   warps 4-11  softmax        : thread = query row, all 128 kv columns of a block; two warpgroups
// The work of a CTA is a sequence of items, a query tile with a kv block each, on two slots of 128 TMEM columns that hold
// S, then P (packed bf16 pairs over the columns that the row's thread has read into registers):
//   two tiles   item i = block i / 2 of tile i % 2; each tile has its own slot and softmax warpgroup
//   one tile    item i = block i on slot i % 2; the first warpgroup takes both slots
// Behind P V of item i the issuer forms S of item i + 2 on the same slot, on the one in-order tensor pipe.
//
// What bounds it: an item costs the tensor cores 2 x 512 clocks, the special-function units 128 x 128 exponentials / 16 =
// 1024, and one warp per scheduler about 1800 from its scores to its probabilities (570 instructions, mostly waiting on one
// another).  With one tile that softmax is the period; with two it runs beside the other tile's products: 1670 clocks an
// item.  40 heads x 16001 causal tokens: 2742 us with one tile per CTA and eight softmax warps on it -> 2060 us (in
// a long run under the power cap 2948 -> 2300); 4 documents of 4096 tokens x 32 heads 91 -> 70 us, 192-wide heads, 3 documents
// x 16 heads 58 -> 44 us.  Measured and not better: 64-row kv blocks with four slots (no tensor work in the chain, 1500
// clocks, but Q is read twice as often: 2180 us, under the cap 2424), sixteen softmax warps (2247), a part of the exponentials
// by polynomial (2100 - 2200), an issuing warp per tile (2090).
//
// The output accumulator is never copied out between blocks.  The running maximum of a row is raised only when the
// new block exceeds it by more than 2^8 in the exponent (probabilities then stay below 256, exact in fp32 sums and
// harmless in bf16); only then the row's accumulator is rescaled in place (tcgen05.ld / multiply / tcgen05.st by the
// softmax warps) before the block's P.V is issued.  The normalisation by the row sum at the end uses the same maximum,
// so the result does not depend on when the maximum was raised.
// Every wait is bounded (mbar_wait): on timeout the role stops, all roles meet at the final barrier,
// TMEM is released and the status word records kernel/site.
//
// Replaces flash-attn 2 `flash_attn_varlen_func` used by the reference (models/modules/attention/interface.py:114-158)
// and produces the optional per-head maximum logit of its TE / FlexAttention providers
// (ops/providers/cuda/attention.py:34-331).
#include "common.cuh"

namespace ttb {

constexpr unsigned KID_ATTN_FWD = 2;
constexpr int AT_BM = 128;   // query rows per tile
constexpr int AT_BN = 128;   // kv rows per block
constexpr int AT_D = 128;    // head dim
constexpr int TILE_BYTES = 128 * 128 * 2;  // one [128 x 128] bf16 tile = two 16 KB swizzle panels
// three warpgroups of 168 registers a thread at launch; the row values of the softmax take more, the issuing warps less
constexpr int AT_THREADS = 384, AT_REGS_ISSUE = 80, AT_REGS_SOFTMAX = 208;
static_assert(AT_REGS_ISSUE + 2 * AT_REGS_SOFTMAX <= 3 * 168, "registers the block was launched with");
constexpr float AT_LAZY = 8.f;             // raise the running maximum only beyond this many powers of two

struct AttnFwdParams {
  const int* q_tiles;   // [n_tiles, 3]: first query row, document start, document end (token indices)
  int tile_rows;        // query rows per table entry: 128 (one tile per CTA) or 256 (two)
  __nv_bfloat16* out;   // [T, Hq, Dv]
  float* lse;           // [Hq, T] natural-log logsumexp of the scaled logits (or null)
  float* max_logit;     // [Hq] per-head maximum scaled logit (atomic max; or null)
  int Hq, Hk;
  int D, Dv;            // width of query / key heads and of value heads
  long long T;
  float scale;          // softmax scale (1/sqrt(D))
  int causal;
};

template <int DQK>
struct AttnSmem {
  // tiles of 128 rows in 64-column swizzle panels of 16 KB, 1024-byte aligned
  static constexpr int QK_BYTES = 128 * DQK * 2;          // one Q or K tile
  static constexpr int KS = DQK == 128 ? 3 : 2;           // K stages
  static constexpr int VS = DQK == 128 ? 2 : 1;           // V stages: what the two Q tiles leave of the 227 KB
  static constexpr int Q = 0;                             // two tiles
  static constexpr int K0 = Q + 2 * QK_BYTES;
  static constexpr int V0 = K0 + KS * QK_BYTES;
  static constexpr int BARS = V0 + VS * TILE_BYTES;
  static constexpr int TOTAL = BARS + 256 + 1024;
  static_assert(VS == 2 || QK_BYTES >= TILE_BYTES, "with one query tile the second V stage lies in the other one's place");
  static constexpr int v_at(int st) { return VS == 1 && st == 1 ? Q + QK_BYTES : V0 + st * TILE_BYTES; }
  static_assert(TOTAL <= 232448, "shared memory of one CTA");
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void atomic_max_float(float* addr, float v) {
  // valid for any sign mix: compare as ordered ints
  if (v >= 0.f) atomicMax(reinterpret_cast<int*>(addr), __float_as_int(v));
  else atomicMin(reinterpret_cast<unsigned int*>(addr), __float_as_uint(v));
}

template <int DQK>
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const AttnFwdParams p) {
  using AttnSmem = ttb::AttnSmem<DQK>;
  constexpr int KS = AttnSmem::KS, VS = AttnSmem::VS, QK_BYTES = AttnSmem::QK_BYTES, NP = DQK / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + AttnSmem::BARS);
  uint64_t* q_full = bars + 0;    // [2 tiles]
  uint64_t* s_full = bars + 2;    // [2 slots] S written; the P V that read this slot before has retired
  uint64_t* p_full = bars + 4;    // [2 slots] P written, O rescaled where a row maximum was raised
  uint64_t* o_step = bars + 6;    // one tile: P V of the next block has retired
  uint64_t* o_full = bars + 18;   // [2 tiles] the last P V of the tile has retired
  uint64_t* k_full = bars + 8;    // [KS]
  uint64_t* k_empty = bars + 11;  // [KS]
  uint64_t* v_full = bars + 14;   // [n_vs]
  uint64_t* v_empty = bars + 16;  // [n_vs]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heads vary fastest in launch order: the tile table lists the tiles with the most KV blocks first, so every head's
  // longest tiles start before any short one, and neighbouring CTAs (the query heads of a group) read the same K / V
  const int entry = blockIdx.y, h = blockIdx.x;
  const int hk = h / (p.Hq / p.Hk);
  const int q0 = p.q_tiles[entry * 3 + 0];
  const int ds = p.q_tiles[entry * 3 + 1];
  const int de = p.q_tiles[entry * 3 + 2];
  // kv blocks of tile t; 0 = no such tile.  Tile 1 sees at least as many blocks as tile 0.
  auto blocks_of = [&](int t) {
    const int q = q0 + t * AT_BM;
    if (t == 1 && (p.tile_rows != 2 * AT_BM || q >= de)) return 0;
    const int kv_end = p.causal ? min(de, q + AT_BM) : de;
    return (kv_end - ds + AT_BN - 1) / AT_BN;
  };
  const int nblk0 = blocks_of(0), nblk1 = blocks_of(1);
  const int nblk = max(nblk0, nblk1);
  const bool two = nblk1 > 0;
  const int n_vs = two ? VS : 2;   // V stages

  if (threadIdx.x == 0) {
    for (int i = 0; i < KS; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&q_full[i], 1); mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&o_full[i], 1);
    }
    mbar_init(o_step, 1);
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
  const uint32_t tm_S = tmem_base;        // 2 slots x 128 columns; P in the first 64 of them: bf16 pairs, column = kv index / 2
  const uint32_t tm_O = tmem_base + 256;  // 2 tiles x 128 columns

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AT_REGS_ISSUE));
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      if (elect_one()) {
        tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
        auto load_q = [&](int t) {
          mbar_expect_tx(&q_full[t], QK_BYTES);
#pragma unroll
          for (int pn = 0; pn < NP; ++pn)
            tma_load_3d(smem + AttnSmem::Q + t * QK_BYTES + pn * 16384, &tmQ, &q_full[t], pn * 64, h, q0 + t * AT_BM);
        };
        auto load_k = [&](int j) -> bool {
          const int ks = j % KS;
          if (!mbar_wait(&k_empty[ks], ((j / KS) & 1) ^ 1, KID_ATTN_FWD, 1)) return false;
          const int kv0 = ds + j * AT_BN;
          mbar_expect_tx(&k_full[ks], QK_BYTES);
#pragma unroll
          for (int pn = 0; pn < NP; ++pn)
            tma_load_3d(smem + AttnSmem::K0 + ks * QK_BYTES + pn * 16384, &tmK, &k_full[ks], pn * 64, hk, kv0);
          return true;
        };
        if (nblk > 0) load_q(0);
        // K runs ahead of V as the scores run ahead of P V: by one block with two tiles, by two with one
        const int ahead = two ? 1 : 2;
        bool ok = nblk > 0 && load_k(0);
        if (two) load_q(1);
        else if (ok && nblk > 1) ok = load_k(1);
        int vs = 0;
        uint32_t vph = 1;
        for (int j = 0; j < nblk && ok; ++j) {
          const int kv0 = ds + j * AT_BN;
          if (two && j + ahead < nblk && !load_k(j + ahead)) break;
          if (!mbar_wait(&v_empty[vs], vph, KID_ATTN_FWD, 2)) break;
          mbar_expect_tx(&v_full[vs], TILE_BYTES);
          tma_load_3d(smem + AttnSmem::v_at(vs), &tmV, &v_full[vs], 0, hk, kv0);
          tma_load_3d(smem + AttnSmem::v_at(vs) + 16384, &tmV, &v_full[vs], 64, hk, kv0);
          if (++vs == n_vs) { vs = 0; vph ^= 1; }
          if (!two && j + ahead < nblk) ok = load_k(j + ahead);
        }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer (the whole warp, see umma_ss_w)
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);  // Q (K-major) x K (K-major)
      const uint32_t idesc_o = make_idesc_bf16(128, (p.Dv + 15) / 16 * 16, false, true);   // P (K-major) x V (MN-major)
      const uint32_t leader = elect_one() ? 1u : 0u;
      const SmemDesc dQ = make_smem_desc2(smem_u32(smem + AttnSmem::Q), 16, 1024);
      const SmemDesc dK = make_smem_desc2(smem_u32(smem + AttnSmem::K0), 16, 1024);
      const SmemDesc dV = make_smem_desc2(smem_u32(smem), 16384, 1024);
      int ks = 0, vs = 0;
      uint32_t kph = 0, vph = 0;
      auto issue_s = [&](int t, int slot) {
        const SmemDesc a = desc_at(dQ, t * QK_BYTES), b = desc_at(dK, ks * QK_BYTES);
#pragma unroll
        for (int kk = 0; kk < DQK / 16; ++kk) {
          const uint32_t off = (kk >> 2) * 16384 + (kk & 3) * 32;
          umma_ss_w(kk * 16 < p.D ? leader : 0u, tm_S + slot * 128, desc_at(a, off), desc_at(b, off), idesc_s, kk != 0);
        }
        umma_commit_w(leader, &s_full[slot]);
      };
      auto wait_k = [&]() { return mbar_wait(&k_full[ks], kph, KID_ATTN_FWD, 4); };
      auto free_k = [&]() {
        umma_commit_w(leader, &k_empty[ks]);
        if (++ks == KS) { ks = 0; kph ^= 1; }
      };
      auto issue_pv = [&](int t, int slot, int j) -> bool {
        if (!mbar_wait(&p_full[slot], (two ? j : j >> 1) & 1, KID_ATTN_FWD, 7)) return false;
        tc_fence_after();
        const SmemDesc b = desc_at(dV, AttnSmem::v_at(vs));
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          // A = P from TMEM: a k-step of 16 kv columns is 8 packed columns
          // B = V: MN-major [kv rows][d], k-step of 16 kv rows = 2048 bytes, d panels 16 KB apart
          umma_ts_w(leader, tm_O + t * 128, tm_S + slot * 128 + kk * 8, desc_at(b, kk * 2048), idesc_o, (j | kk) != 0);
        }
        if (!two) umma_commit_w(leader, o_step);
        if (j + 1 == (t == 0 ? nblk0 : nblk1)) umma_commit_w(leader, &o_full[t]);
        return true;
      };
      bool ok = nblk > 0 && wait_k() && mbar_wait(&q_full[0], 0, KID_ATTN_FWD, 3);
      if (ok) {
        issue_s(0, 0);
        if (two) {
          ok = mbar_wait(&q_full[1], 0, KID_ATTN_FWD, 3);
          if (ok) issue_s(1, 1);
        }
        free_k();
        if (ok && !two && nblk > 1) {
          ok = wait_k();
          if (ok) issue_s(0, 1);
          free_k();
        }
      }
      for (int j = 0; j < nblk && ok; ++j) {
        if (!mbar_wait(&v_full[vs], vph, KID_ATTN_FWD, 6)) break;
        const bool more = j + (two ? 1 : 2) < nblk;
        if (more && !wait_k()) break;
        if (two) {
          if (j < nblk0) {
            ok = issue_pv(0, 0, j);
            if (!ok) break;
            if (j + 1 < nblk0) issue_s(0, 0);
          }
          ok = issue_pv(1, 1, j);
          if (!ok) break;
          if (more) issue_s(1, 1);
        } else {
          ok = issue_pv(0, j & 1, j);
          if (!ok) break;
          if (more) issue_s(0, j & 1);
        }
        // committed behind everything issued above, where a later block waits for it: behind the last product of the tiles nothing
        // may be left that signals a barrier, or it could arrive when the CTA has ended
        if (j + n_vs < nblk) umma_commit_w(leader, &v_empty[vs]);
        if (++vs == n_vs) { vs = 0; vph ^= 1; }
        if (more) free_k();
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(AT_REGS_SOFTMAX));
    // ---------------------------------------------------------------- softmax (thread = query row of tile t)
    const int t = (warp - 4) >> 2;
    const int n = t == 0 ? nblk0 : nblk1;
    const int lg = warp & 3;
    const int row = lg * 32 + lane;
    const int qt = q0 + t * AT_BM;
    const int qrow = qt + row;
    const bool row_ok = qrow < de;
    const float c = p.scale * 1.4426950408889634f;
    const uint32_t lane_off = static_cast<uint32_t>(lg * 32) << 16;
    const uint32_t t_O = tm_O + t * 128 + lane_off;
    float m_run = -INFINITY, l_run = 0.f, mx_logit = -INFINITY;
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      const int slot = two ? t : j & 1;
      const uint32_t t_S = tm_S + slot * 128 + lane_off;
      if (!mbar_wait(&s_full[slot], (two ? j : j >> 1) & 1, KID_ATTN_FWD, 9)) { ok = false; break; }
      tc_fence_after();
      float s[128];
      {
        uint32_t va[32], vb[32], vc[32], vd[32];
        tmem_ld_32x32b_x32(t_S, va);
        tmem_ld_32x32b_x32(t_S + 32, vb);
        tmem_ld_32x32b_x32(t_S + 64, vc);
        tmem_ld_32x32b_x32(t_S + 96, vd);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          s[i] = __uint_as_float(va[i]);
          s[32 + i] = __uint_as_float(vb[i]);
          s[64 + i] = __uint_as_float(vc[i]);
          s[96 + i] = __uint_as_float(vd[i]);
        }
      }
      const int kv0 = ds + j * AT_BN;
      if ((kv0 + AT_BN > de) || (p.causal && kv0 + AT_BN - 1 > qt)) {
        // columns of this block that the row sees: [0, lim)
        const int lim = row_ok ? (p.causal ? min(de - 1, qrow) : de - 1) - kv0 + 1 : 0;
#pragma unroll
        for (int i = 0; i < 128; ++i) s[i] = i < lim ? s[i] : -INFINITY;
      }
      float m0 = s[0], m1 = s[1], m2 = s[2], m3 = s[3];
#pragma unroll
      for (int i = 4; i + 8 <= 128; i += 8) {
        m0 = fmax3(m0, s[i], s[i + 1]);
        m1 = fmax3(m1, s[i + 2], s[i + 3]);
        m2 = fmax3(m2, s[i + 4], s[i + 5]);
        m3 = fmax3(m3, s[i + 6], s[i + 7]);
      }
      m0 = fmax3(m0, s[124], s[125]);
      m1 = fmax3(m1, s[126], s[127]);
      const float m_blk = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
      mx_logit = fmaxf(mx_logit, m_blk);
      // raise the running maximum only when the block exceeds it by more than AT_LAZY powers of two
      float alpha = 1.f;
      if (m_blk > m_run && (m_run == -INFINITY || (m_blk - m_run) * c > AT_LAZY)) {
        alpha = (m_run == -INFINITY) ? 0.f : fast_exp2((m_run - m_blk) * c);
        m_run = m_blk;
      }
      const float mc = (m_run == -INFINITY) ? 0.f : m_run * c;
      // O_t may only be touched once its last P V has retired (rare: only when a row maximum was raised).  With two tiles the
      // scores of this block were formed behind that product, with one behind the product of the block before it.
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        if (!two && !mbar_wait(o_step, (j - 1) & 1, KID_ATTN_FWD, 10)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int cb = 0; cb < 8; ++cb) {
          uint32_t v[16];
          tmem_ld_32x32b_x16(t_O + cb * 16, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
          tmem_st_32x32b_x16(t_O + cb * 16, v);
        }
      }
      // two columns per instruction: exponent argument, row-sum accumulation (of the unrounded probabilities)
      const uint64_t cc = f2_pack(c, c), nmc = f2_pack(-mc, -mc);
      uint64_t la = f2_pack(0.f, 0.f), lb = la;
#pragma unroll
      for (int qb = 0; qb < 4; ++qb) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float a0, a1;
          f2_unpack(f2_fma(f2_pack(s[qb * 32 + 2 * i], s[qb * 32 + 2 * i + 1]), cc, nmc), a0, a1);
          const float e0 = fast_exp2(a0), e1 = fast_exp2(a1);
          w[i] = pack_bf16(e0, e1);
          if (i & 1) lb = f2_add(lb, f2_pack(e0, e1));
          else la = f2_add(la, f2_pack(e0, e1));
        }
        tmem_st_32x32b_x16(t_S + qb * 16, w);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[slot]);
      float l_lo, l_hi;
      f2_unpack(f2_add(la, lb), l_lo, l_hi);
      l_run = l_run * alpha + (l_lo + l_hi);
    }
    // ---- epilogue
    if (n > 0) {
      if (ok) ok = mbar_wait(&o_full[t], 0, KID_ATTN_FWD, 11);
      if (ok && row_ok && p.lse)
        p.lse[static_cast<long long>(h) * p.T + qrow] = (l_run > 0.f) ? m_run * p.scale + logf(l_run) : -INFINITY;
      if (p.max_logit) {
        const float wm = warp_max(row_ok ? mx_logit * p.scale : -INFINITY);
        if (lane == 0 && wm > -INFINITY) atomic_max_float(&p.max_logit[h], wm);
      }
      if (ok) {
        tc_fence_after();
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        __nv_bfloat16* dst = p.out + (static_cast<long long>(qrow) * p.Hq + h) * p.Dv;
#pragma unroll
        for (int cb = 0; cb < 4; ++cb) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(t_O + cb * 32, v);
          tmem_ld_wait();
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              if (cb * 32 + i >= p.Dv) continue;
              uint4 w;
              w.x = pack_bf16(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv);
              w.y = pack_bf16(__uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv);
              w.z = pack_bf16(__uint_as_float(v[i + 4]) * inv, __uint_as_float(v[i + 5]) * inv);
              w.w = pack_bf16(__uint_as_float(v[i + 6]) * inv, __uint_as_float(v[i + 7]) * inv);
              *reinterpret_cast<uint4*>(dst + cb * 32 + i) = w;
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int DQK>
static int launch_attn_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnFwdParams& p, int n_tiles,
                           cudaStream_t stream) {
  static bool smem_done[16] = {};
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(attn_fwd_kernel<DQK>), AttnSmem<DQK>::TOTAL, smem_done);
  if (e != cudaSuccess) return 300 + static_cast<int>(e);
  dim3 grid(p.Hq, n_tiles);
  attn_fwd_kernel<DQK><<<grid, AT_THREADS, AttnSmem<DQK>::TOTAL, stream>>>(tq, tk, tv, p);
  return 0;
}

}  // namespace ttb

using namespace ttb;

// q: [T, Hq, D] (row stride ldq), k: [T, Hk, D] (ldk), v: [T, Hk, Dv] (ldv; may be a strided view), out: [T, Hq, Dv]; D and Dv up
// to 128 in multiples of 8, or D = 192 with Dv = 128
TTB_EXPORT int ttb_attn_fwd(const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv,
                            void* out, float* lse, float* max_logit, const int* q_tiles, int n_tiles, int tile_rows, long long T,
                            int Hq, int Hk, int D, int Dv, float scale, int causal, void* stream) {
  if (D < 8 || Dv < 8 || D % 8 || Dv % 8 || Dv > AT_D || (D > 128 && !(D == 192 && Dv == AT_D)) || Hq % Hk) return 901;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8)) return 902;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out)) & 15)
    return 903;
  if (tile_rows != 128 && tile_rows != 256) return 904;
  if (n_tiles == 0) return 0;
  CUtensorMap tq, tk, tv;
  if (make_heads_map(&tq, q, T, ldq, Hq, D, AT_BM)) return 101;
  if (make_heads_map(&tk, k, T, ldk, Hk, D, AT_BN)) return 102;
  if (make_heads_map(&tv, v, T, ldv, Hk, Dv, AT_BN)) return 103;
  AttnFwdParams p{q_tiles, tile_rows, (__nv_bfloat16*)out, lse, max_logit, Hq, Hk, D, Dv, T, scale, causal};
  const int rc = D <= 128 ? launch_attn_fwd<128>(tq, tk, tv, p, n_tiles, reinterpret_cast<cudaStream_t>(stream))
                          : launch_attn_fwd<192>(tq, tk, tv, p, n_tiles, reinterpret_cast<cudaStream_t>(stream));
  if (rc) return rc;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

TTB_EXPORT int ttb_attn_status(unsigned int* out4, int reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out4, ttb::g_status_word, sizeof(unsigned int) * 4);
  if (e != cudaSuccess) return (int)e;
  if (reset) {
    unsigned int z[4] = {0, 0, 0, 0};
    e = cudaMemcpyToSymbol(ttb::g_status_word, z, sizeof(z));
  }
  return (int)e;
}
