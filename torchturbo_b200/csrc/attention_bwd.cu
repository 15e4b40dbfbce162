// Variable-length flash attention backward for sm_100a (GQA, causal or full; heads up to 128 wide in multiples of 8, or value
// heads 128 wide with query / key heads 192 for multi-head latent attention).  The kernel is built in two forms: with the dQ^T product and its
// reduction (128-wide heads, the default), and without it, where dQ comes from the query-major pass in
// attention_bwd_dq.cu (192-wide heads, whose accumulators do not fit tensor memory together, and the bit-reproducible
// mode of 128-wide heads).
//
// One CTA owns one 128-row KV tile of one document for one *query* head; K_j and V_j stay resident in shared memory
// and dK_j / dV_j accumulate in TMEM over every 64-row query tile that can see the KV tile.  With grouped-query
// attention the CTAs of the query heads that share a KV head add their dK / dV into fp32 accumulators by TMA reductions
// (splitting by query head keeps the longest CTA short: a causal KV tile near the start of a long document
// is seen by every later query tile).  Per query-tile iteration, all on tcgen05 with M = 128:
//     S^T  = K_j  Q_i^T          [kv, q]     (K-major  x K-major)
//     dP^T = V_j  dO_i^T         [kv, q]     (K-major  x K-major)
//     P^T  = exp2(S^T c - lse_q),  dS^T = P^T (dP^T - Delta_q) scale        (one thread per kv row, P -> TMEM, dS -> smem)
//     dV  += P^T  dO_i           [kv, d]     (TMEM     x MN-major)
//     dK  += dS^T Q_i            [kv, d]     (K-major  x MN-major)
//     dQ^T = K_j^T dS^T          [d, q]      (MN-major x MN-major)  -> transposed through shared memory and added
//                                            into the fp32 dQ buffer by one TMA reduction per tile (the L2 does the adds)
// Warp roles: 0 TMA producer, 1 MMA issuer, 2-9 softmax/dS, 10-13 dQ read-out.  The softmax of a tile is the longest
// dependent chain of an iteration (TMEM read, 64 exponentials per kv row, two bf16 tiles to shared memory), so two
// warpgroups share it: warps 2-5 take query columns 0-31 of every kv row, warps 6-9 columns 32-63 (a warp may read
// the TMEM lanes 32 (warp % 4) .. +31 at any column).  P^T (TMEM) and dS^T (shared memory; one buffer with 192-wide heads) are
// double-buffered: the softmax warps of query tile i+1 run while the tensor cores still consume the P^T / dS^T of tile i, and the
// dQ read-out of tile i overlaps the products of tile i+1.  Waits are bounded; on timeout the roles drain to the final
// barrier, TMEM is freed and the status word records where the wait gave up.
//
// What bounds it: 2300 clocks per pair of tiles, of which the products need 1280 at the tensor rate and 1500 with the 192 KB that
// they read through shared memory (another 112 KB are written and read by the other roles); the softmax warps' chain is 1800.  It
// was 3300: P^T in shared memory left room for two Q / dO stages only, whose refill was waited for (700); the row statistics were
// waited for at the top of every iteration (700); masks and dS stores between the exponentials kept them from overlapping; and
// every CTA ended with 9700 clocks of 16-byte atomics (7500 now, all of it traffic of 128 KB of sums).  Whole call in us, before ->
// now: 4096 tokens in four documents, 32 / 4 heads 355 -> 296, bit-reproducible 703 -> 475; 8192 tokens, 32 / 8 heads 1070 -> 893;
// 192 / 128-wide heads, 4096 x 16 295 -> 245; five documents of 600, 16 heads of 72, full attention 101 -> 89; 300 x 8 29 -> 26.
//
// Replaces flash-attn 2's backward used through the reference attention interface
// (models/modules/attention/interface.py:114-158).
#include "common.cuh"
#include <type_traits>

namespace ttb {

constexpr unsigned KID_ATTN_BWD = 4;
constexpr int BW_KV = 128;   // kv rows per CTA
constexpr int BW_Q = 64;     // query rows per iteration
constexpr int BW_D = 128;

struct AttnBwdParams {
  const int* kv_tiles;   // [n_tiles, 3]: first kv row, document start, document end
  const float* lse;      // [Hq, T]
  const float* delta;    // [Hq, T]  rowsum(dO * O)
  float* dq_acc;         // [T, Hq, D] fp32, zero before the kernel
  __nv_bfloat16* dk;     // [T, Hk, D]   written directly when Hq == Hk
  __nv_bfloat16* dv;     // [T, Hk, D]
  float* dk_acc;         // [T, Hk, D] fp32, zero before the kernel (used when Hq > Hk)
  float* dv_acc;
  int Hq, Hk;
  int D, Dv;             // width of query / key heads and of value heads
  long long T;
  float scale;
  int causal;
  int group_loop;   // 1: one CTA per kv head loops over the query heads of its group (no atomics on dK / dV)
};

template <int DQK, bool WITH_DQ>
struct BwdSmem {
  static constexpr int K_BYTES = 128 * DQK * 2;     // K tile: DQK / 64 panels of 16 KB
  static constexpr int Q_BYTES = 64 * DQK * 2;      // Q tile: DQK / 64 panels of 8 KB
  static constexpr int STAGES = 3;                  // Q / dO tiles on their way or in use
  static constexpr int DS_BUFS = DQK == 128 ? 2 : 1;
  static constexpr int K = 0;
  static constexpr int V = K + K_BYTES;             // 32 KB
  static constexpr int Q0 = V + 32768;
  static constexpr int DO0 = Q0 + STAGES * Q_BYTES;
  static constexpr int DST = DO0 + STAGES * 16384;  // 16 KB each: dS^T [128 kv][64 q]
  static constexpr int DQS = DST + DS_BUFS * 16384; // 32 KB  dQ tile [64 q][128 d] fp32, source of the TMA reduction
  static constexpr int STAT = DQS + (WITH_DQ ? 32768 : 0);  // float [2][lse, delta][128]: two iterations' rows, two buffers
  static constexpr int BARS = STAT + 2 * 2 * 128 * 4;
  static constexpr int TOTAL = BARS + 256;
  static_assert(TOTAL <= 232448, "one CTA per SM");
  static_assert(DST >= 8 * 16384, "the tiles before dS^T hold dK and dV in fp32 at the end");
};

__device__ __forceinline__ float bw_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two pairs of fp32 from shared memory; volatile without a memory clobber: stays behind the waits, free among the arithmetic
__device__ __forceinline__ void ld_shared_pairs(uint32_t addr, uint64_t& a, uint64_t& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}

// Warp-collective: 32 consecutive fp32 columns of two accumulators, both loads in flight before the one wait.
__device__ __forceinline__ void tmem_ld32x2(uint32_t ta, uint32_t tb, float (&a)[32], float (&b)[32]) {
  uint32_t va[32], vb[32];
  tmem_ld_32x32b_x32(ta, va);
  tmem_ld_32x32b_x32(tb, vb);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    a[i] = __uint_as_float(va[i]);
    b[i] = __uint_as_float(vb[i]);
  }
}

// Warp-collective: 64 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, float (&out)[64]) {
#pragma unroll
  for (int cb = 0; cb < 2; ++cb) {
    uint32_t v[32];
    tmem_ld_32x32b_x32(taddr + cb * 32, v);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) out[cb * 32 + i] = __uint_as_float(v[i]);
  }
}

// FULL: heads as wide as the tiles (widths known at compile time, two-dimensional maps).  With the widths as variables and
// three-dimensional maps the 128-wide case (4096 tokens, 32 / 8 heads) took 269 us instead of 257.
template <int DQK, bool WITH_DQ, bool FULL>
__global__ void __launch_bounds__(448, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV,
                const AttnBwdParams p) {
  static_assert(DQK == 128 || !WITH_DQ, "the fused dQ path exists for 128-wide heads only");
  using BwdSmem = ttb::BwdSmem<DQK, WITH_DQ>;
  const int D = FULL ? DQK : p.D, Dv = FULL ? BW_D : p.Dv;
  auto load_head = [](void* dst, const CUtensorMap* map, uint64_t* bar, int col, int head, int width, int row) {
    if (FULL) tma_load_2d(dst, map, bar, head * width + col, row);
    else tma_load_3d(dst, map, bar, col, head, row);
  };
  constexpr int NP = DQK / 64, Q_BYTES = BwdSmem::Q_BYTES;
  extern __shared__ __align__(1024) uint8_t smem[];      // swizzled tiles; there is no room to align them by hand
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) set_status(KID_ATTN_BWD, 12, blockIdx.x);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BwdSmem::BARS);
  uint64_t* kv_full = bars + 0;
  constexpr int STAGES = BwdSmem::STAGES;
  uint64_t* qdo_full = bars + 1;    // [3]
  uint64_t* qdo_empty = bars + 4;   // [3]
  uint64_t* st_full = bars + 7;
  uint64_t* st_empty = bars + 8;
  uint64_t* pds_full = bars + 9;    // [2]
  uint64_t* pds_empty = bars + 11;  // [2]
  uint64_t* dq_full = bars + 13;
  uint64_t* dq_empty = bars + 14;
  uint64_t* acc_full = bars + 15;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* s_dead = reinterpret_cast<volatile int*>(bars + 17);   // a softmax warp's wait gave up
  volatile int* s_dead_dq = reinterpret_cast<volatile int*>(bars + 18);  // a dQ warp's wait gave up
  float* s_stat = reinterpret_cast<float*>(smem + BwdSmem::STAT);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Launch order.  With dQ in this kernel, tiles vary fastest: the CTAs of one head run together and share its Q / dO
  // rows in the L2 (with heads fastest the 64K-token backward was 12 % slower).  Without dQ (the query-major pass
  // follows), heads vary fastest as in the forward kernel, so the longest tiles of every head start first: measured
  // 10 % faster at 8192 tokens, equal at 65536.
  const int tile = WITH_DQ ? blockIdx.x : blockIdx.y;
  const int head = WITH_DQ ? blockIdx.y : blockIdx.x;
  const int G = p.Hq / p.Hk;
  // default: one CTA per query head (parallel, dK / dV of a group summed with atomics); group loop: one CTA per kv head
  // walks the query heads of its group one after the other and owns dK / dV alone
  const int hk = p.group_loop ? head : head / G;
  const int hq = p.group_loop ? hk * G : head;
  const int kv0 = p.kv_tiles[tile * 3 + 0];
  const int ds = p.kv_tiles[tile * 3 + 1];
  const int de = p.kv_tiles[tile * 3 + 2];
  // query tiles (64 rows, aligned to the document start) that can see this kv tile
  const int q_first = p.causal ? ds + ((kv0 - ds) / BW_Q) * BW_Q : ds;
  const int n_qt = (de - q_first + BW_Q - 1) / BW_Q;
  const int n_it = p.group_loop ? n_qt * G : n_qt;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < STAGES; ++i) { mbar_init(&qdo_full[i], 1); mbar_init(&qdo_empty[i], 1); }
    mbar_init(st_full, 1); mbar_init(st_empty, 8);
    for (int i = 0; i < 2; ++i) { mbar_init(&pds_full[i], 8); mbar_init(&pds_empty[i], 1); }
    mbar_init(dq_full, 1); mbar_init(dq_empty, 4);
    mbar_init(acc_full, 1);
    *s_dead = 0;
    *s_dead_dq = 0;
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
  const uint32_t tm_ST = tmem_base;          // 64 cols
  const uint32_t tm_DPT = tmem_base + 64;    // 64 cols
  const uint32_t tm_PT = tmem_base + 128;    // 2 x 32 cols: P^T as packed bf16, the A operand of dV
  const uint32_t tm_DQT = tmem_base + 192;   // 64 cols (form with dQ)
  const uint32_t tm_DV = tmem_base + (WITH_DQ ? 256 : 192);    // 128 cols
  const uint32_t tm_DK = tmem_base + (WITH_DQ ? 384 : 320);    // DQK cols

  auto it_head = [&](int it) { return p.group_loop ? hq + it / n_qt : hq; };
  auto it_q0 = [&](int it) { return q_first + (p.group_loop ? it % n_qt : it) * BW_Q; };

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
      mbar_expect_tx(kv_full, BwdSmem::K_BYTES + 32768);
#pragma unroll
      for (int pn = 0; pn < NP; ++pn) load_head(smem + BwdSmem::K + pn * 16384, &tmK, kv_full, pn * 64, hk, DQK, kv0);
      load_head(smem + BwdSmem::V, &tmV, kv_full, 0, hk, 128, kv0);
      load_head(smem + BwdSmem::V + 16384, &tmV, kv_full, 64, hk, 128, kv0);
      int st = 0;
      uint32_t ph = 0;
      for (int it = 0; it < n_it; ++it) {
        if (!mbar_wait(&qdo_empty[st], ph ^ 1, KID_ATTN_BWD, 1)) break;
        const int h = it_head(it), q0 = it_q0(it);
        mbar_expect_tx(&qdo_full[st], Q_BYTES + 16384);
        uint8_t* sq = smem + BwdSmem::Q0 + st * Q_BYTES;
        uint8_t* sd = smem + BwdSmem::DO0 + st * 16384;
#pragma unroll
        for (int pn = 0; pn < NP; ++pn) load_head(sq + pn * 8192, &tmQ, &qdo_full[st], pn * 64, h, DQK, q0);
        load_head(sd, &tmDO, &qdo_full[st], 0, h, 128, q0);
        load_head(sd + 8192, &tmDO, &qdo_full[st], 64, h, 128, q0);
        if (++st == STAGES) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (the whole warp, see umma_ss_w)
    // One diverged lane took long enough over the descriptors to hold up the tensor cores: 4096 tokens, 32 / 8 heads, four
    // documents 268 -> 260 us; 192-wide heads 207 -> 199; 8192 tokens, 32 heads 1772 -> 1700.
    {
      constexpr uint32_t id_s = make_idesc_bf16(128, 64, false, false);
      const uint32_t id_acc = make_idesc_bf16(128, (Dv + 15) / 16 * 16, false, true);
      const uint32_t id_dk = make_idesc_bf16(128, (D + 15) / 16 * 16, false, true);
      constexpr uint32_t id_dq = make_idesc_bf16(128, 64, true, true);
      const uint32_t leader = elect_one() ? 1u : 0u;
      // operands read along their rows (K-major) and, where a product reduces over rows, across them (MN-major)
      const SmemDesc dK = make_smem_desc2(smem_u32(smem + BwdSmem::K), 16, 1024), dV = make_smem_desc2(smem_u32(smem + BwdSmem::V), 16, 1024);
      const SmemDesc dQ = make_smem_desc2(smem_u32(smem + BwdSmem::Q0), 16, 1024), dDO = make_smem_desc2(smem_u32(smem + BwdSmem::DO0), 16, 1024);
      const SmemDesc dDST = make_smem_desc2(smem_u32(smem + BwdSmem::DST), 16, 1024);
      const SmemDesc dKt = make_smem_desc2(smem_u32(smem + BwdSmem::K), 16384, 1024), dDSt = make_smem_desc2(smem_u32(smem + BwdSmem::DST), 8192, 1024);
      const SmemDesc dQt = make_smem_desc2(smem_u32(smem + BwdSmem::Q0), 8192, 1024), dDOt = make_smem_desc2(smem_u32(smem + BwdSmem::DO0), 8192, 1024);
      bool ok = mbar_wait(kv_full, 0, KID_ATTN_BWD, 2);
      int st_s = 0, st = 0;          // stage of the tile whose scores are formed / whose gradients are
      uint32_t ph_s = 0;
      auto issue_scores = [&](int it) -> bool {
        const int st = st_s;
        const uint32_t ph = ph_s;
        if (++st_s == STAGES) { st_s = 0; ph_s ^= 1; }
        if (!mbar_wait(&qdo_full[st], ph, KID_ATTN_BWD, 3)) return false;
        if (!mbar_wait(st_empty, (it & 1) ^ 1, KID_ATTN_BWD, 4)) return false;
        tc_fence_after();
        const SmemDesc q = desc_at(dQ, st * Q_BYTES), d_o = desc_at(dDO, st * 16384);
#pragma unroll
        for (int kk = 0; kk < DQK / 16; ++kk) {  // reduction over the query / key head width
          const uint32_t offa = (kk >> 2) * 16384 + (kk & 3) * 32;   // K / V tiles: [128 rows][64 d] panels
          const uint32_t offb = (kk >> 2) * 8192 + (kk & 3) * 32;    // Q / dO tiles: [64 rows][64 d] panels
          umma_ss_w(kk * 16 < D ? leader : 0u, tm_ST, desc_at(dK, offa), desc_at(q, offb), id_s, kk != 0);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t offa = (kk >> 2) * 16384 + (kk & 3) * 32;
          const uint32_t offb = (kk >> 2) * 8192 + (kk & 3) * 32;
          umma_ss_w(kk * 16 < Dv ? leader : 0u, tm_DPT, desc_at(dV, offa), desc_at(d_o, offb), id_s, kk != 0);
        }
        umma_commit_w(leader, st_full);
        return true;
      };
      if (ok && n_it > 0) ok = issue_scores(0);
      for (int it = 0; it < n_it && ok; ++it) {
        if (it + 1 < n_it) {
          if (!issue_scores(it + 1)) { ok = false; break; }
        }
        const int b = it & 1, db = it % BwdSmem::DS_BUFS;
        if (!mbar_wait(&pds_full[b], (it >> 1) & 1, KID_ATTN_BWD, 5)) { ok = false; break; }
        tc_fence_after();
        const SmemDesc dst = desc_at(dDST, db * 16384), dst_t = desc_at(dDSt, db * 16384);
        const SmemDesc q_t = desc_at(dQt, st * Q_BYTES), do_t = desc_at(dDOt, st * 16384);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {  // reduction over q = 64
          // A: P^T from tensor memory (16 queries are 8 columns), dS^T K-major single panel; B: dO / Q as [q rows][d] MN-major, d
          // panels 8 KB apart
          umma_ts_w(leader, tm_DV, tm_PT + b * 32 + kk * 8, desc_at(do_t, kk * 2048), id_acc, (it | kk) != 0);
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          umma_ss_w(leader, tm_DK, desc_at(dst, kk * 32), desc_at(q_t, kk * 2048), id_dk, (it | kk) != 0);
        }
        umma_commit_w(leader, &qdo_empty[st]);
        if (++st == STAGES) st = 0;
        if (WITH_DQ) {
          if (!mbar_wait(dq_empty, (it & 1) ^ 1, KID_ATTN_BWD, 6)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {  // reduction over kv = 128
            // A: K^T from the K tile ([kv rows][d], MN-major, d panels 16 KB apart); B: dS^T ([kv rows][q]) MN-major
            umma_ss_w(leader, tm_DQT, desc_at(dKt, kk * 2048), desc_at(dst_t, kk * 2048), id_dq, kk != 0);
          }
          umma_commit_w(leader, dq_full);
        }
        umma_commit_w(leader, &pds_empty[b]);
      }
      if (ok) umma_commit_w(leader, acc_full);
    }
  } else if (warp < 10) {
    // ---------------------------------------------------------------- softmax / dS (thread = kv row, 32 query columns)
    const int lg = warp & 3;
    const int half = (warp - 2) >> 2;          // 0: query columns 0-31, 1: columns 32-63
    const int row = lg * 32 + lane;
    const int kv = kv0 + row;
    const bool kv_ok = kv < de;
    const float c = p.scale * 1.4426950408889634f;
    const int tid = threadIdx.x - 64;  // 0..255 inside the two groups
    bool ok = true;
    // lse / delta of the 128 query rows of two iterations are staged two iterations ahead, one value a thread (double-buffered).  The
    // load is issued before the two and its value is touched only after them: with the factors applied where it was loaded, every
    // iteration began with the load's latency, a third of its time.
    const int srow = tid & 127;
    const bool is_lse = tid < 128;
    const float* stat = is_lse ? p.lse : p.delta;
    int h_n = hq, q0_n = q_first;              // head and first query row of the iteration to be staged or done next
    auto advance = [&](int& h, int& q0) {
      q0 += BW_Q;
      if (q0 >= de) { q0 = q_first; ++h; }
    };
    int q_mine = 0;                            // this thread's row of the two iterations that are staged
    auto fetch = [&](int h, int q0) {          // the second one may lie past the last iteration: its rows are loaded and not used
      if (srow >= 64) advance(h, q0);
      q_mine = q0 + (srow & 63);
      float v;                                 // volatile: the compiler would move a plain load down to the use of its value
      asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(stat + static_cast<long long>(min(h, p.Hq - 1)) * p.T + min(q_mine, de - 1)));
      return v;
    };
    auto put = [&](int pair, float v) {
      const bool in = q_mine < de;
      s_stat[(pair & 1) * 256 + tid] = is_lse ? (in ? -v * 1.4426950408889634f : -INFINITY) : (in ? -v * p.scale : 0.f);
    };
    put(0, fetch(h_n, q0_n));
    asm volatile("bar.sync 1, 256;" ::: "memory");
    // one iteration; false when a wait gave up (the caller still joins the group barrier, so no warp is left in it)
    auto body = [&](int it) -> bool {
      const int q0 = q0_n;
      advance(h_n, q0_n);
      if (!mbar_wait(st_full, it & 1, KID_ATTN_BWD, 7)) return false;
      tc_fence_after();
      float s[32], dp[32];
      const uint32_t lane_off = (static_cast<uint32_t>(lg * 32) << 16) + half * 32;
      tmem_ld32x2(tm_ST + lane_off, tm_DPT + lane_off, s, dp);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(st_empty);
      const uint32_t lse = smem_u32(s_stat) + (((it >> 1) & 1) * 256 + (it & 1) * 64 + half * 32) * 4, dl = lse + 512;
      const int qh = q0 + half * 32;
      const bool need_mask = (q0 + BW_Q > de) || (kv0 + BW_KV > de) || (p.causal && kv0 + BW_KV - 1 > qh);
      // The tiles that used these buffers must have been consumed: P^T two iterations ago (a fresh barrier passes), and dS^T, where
      // it has one buffer, by the iteration before, whose products were issued before the scores of this one were read.
      if (!mbar_wait(&pds_empty[it & 1], ((it >> 1) & 1) ^ 1, KID_ATTN_BWD, 8)) return false;
      if (BwdSmem::DS_BUFS == 1 && it > 0 && !mbar_wait(&pds_empty[(it - 1) & 1], ((it - 1) >> 1) & 1, KID_ATTN_BWD, 11)) return false;
      tc_fence_after();
      // two columns per instruction; the staged row statistics are -lse log2(e) and -Delta scale
      const uint64_t cc = f2_pack(c, c), sc2 = f2_pack(p.scale, p.scale);
      uint32_t wp[16], wd[16];
      // Masked tiles have their own copy (a branch around every pair of columns kept their chains of exponential, product and
      // conversion from overlapping), and dS is stored behind all of them for the same reason.
      auto columns = [&](auto masked) {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          uint64_t lv[4], dlv[4];
          ld_shared_pairs(lse + ch * 32, lv[0], lv[1]);
          ld_shared_pairs(lse + ch * 32 + 16, lv[2], lv[3]);
          ld_shared_pairs(dl + ch * 32, dlv[0], dlv[1]);
          ld_shared_pairs(dl + ch * 32 + 16, dlv[2], dlv[3]);
#pragma unroll
          for (int qq = 0; qq < 4; ++qq) {
            const int col = ch * 8 + qq * 2;
            float a0, a1;
            f2_unpack(f2_fma(f2_pack(s[col], s[col + 1]), cc, lv[qq]), a0, a1);
            float p0 = bw_exp2(a0), p1 = bw_exp2(a1);
            if (decltype(masked)::value) {
              const int q = qh + col;
              p0 = (kv_ok && q < de && (!p.causal || kv <= q)) ? p0 : 0.f;
              p1 = (kv_ok && q + 1 < de && (!p.causal || kv <= q + 1)) ? p1 : 0.f;
            }
            float d0, d1;
            f2_unpack(f2_mul(f2_pack(p0, p1), f2_fma(f2_pack(dp[col], dp[col + 1]), sc2, dlv[qq])), d0, d1);
            wp[ch * 4 + qq] = pack_bf16(p0, p1);
            wd[ch * 4 + qq] = pack_bf16(d0, d1);
          }
        }
      };
      if (need_mask) columns(std::true_type{});
      else columns(std::false_type{});
      const uint32_t ds_row = smem_u32(smem + BwdSmem::DST) + (it % BwdSmem::DS_BUFS) * 16384 + row * 128;
#pragma unroll
      for (int ch = 0; ch < 4; ++ch)
        st_shared_v4(ds_row + (((half * 4 + ch) ^ (row & 7)) * 16), wd[4 * ch], wd[4 * ch + 1], wd[4 * ch + 2], wd[4 * ch + 3]);
      tmem_st_32x32b_x16(tm_PT + (it & 1) * 32 + half * 16 + (static_cast<uint32_t>(lg * 32) << 16), wp);
      tmem_st_wait();
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pds_full[it & 1]);
      return true;
    };
    for (int it = 0; it < n_it; it += 2) {
      int h_2 = h_n, q0_2 = q0_n;
      advance(h_2, q0_2);
      advance(h_2, q0_2);
      const float staged = fetch(h_2, q0_2);   // past the last iteration too: some row of this head
      if (!body(it) || (it + 1 < n_it && !body(it + 1))) { *s_dead = 1; ok = false; }
      put((it >> 1) + 1, staged);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (*s_dead) { ok = false; break; }
    }
    // ---- epilogue: dV (columns 0-31 group) or dK (the other) of this warp's 32 kv rows, by way of shared memory and the copy engine.
    // All products have retired, so that K, V and the Q / dO stages are free: 16 KB per warp.  The rows lie kilobytes apart in
    // memory, and a thread that adds its own row 16 bytes at a time held the CTA up for 9700 clocks.
    if (ok) ok = mbar_wait(acc_full, 0, KID_ATTN_BWD, 9);       // a kv tile is seen by its own rows at least
    if (ok) {
      tc_fence_after();
      const int which = half, width = which == 0 ? Dv : D;
      const CUtensorMap* map = which == 0 ? &tmDV : &tmDK;
      const uint32_t tm = (which == 0 ? tm_DV : tm_DK) + (static_cast<uint32_t>(lg * 32) << 16);
      const int row0 = kv0 + lg * 32;
      const bool sums = G > 1 && !p.group_loop;
      uint8_t* tile = smem + (which * 4 + lg) * 16384;
      if (sums) {
        // fp32, 32 columns a box; rows past the document are other documents', to which zeros are added
#pragma unroll 1
        for (int cb = 0; cb * 32 < width; ++cb) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tm + cb * 32, v);
          tmem_ld_wait();
          uint8_t* box = tile + (cb & 3) * 4096;
          if (cb == 4) {                        // 192-wide heads: the first boxes once more
            if (lane == 0) bulk_wait_read_all();
            __syncwarp();
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            uint4 w = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            if (!kv_ok) w = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(box + lane * 128 + ((i ^ (lane & 7)) << 4)) = w;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (FULL) tma_reduce_add_2d(map, box, hk * width + cb * 32, row0);
            else tma_reduce_add_3d(map, box, cb * 32, hk, row0);
            bulk_commit_group();
          }
        }
      } else {
        const bool whole = row0 + 32 <= de;     // no row of another document, which its own CTA writes
#pragma unroll 1
        for (int cb = 0; cb * 64 < width; ++cb) {
          uint32_t v[2][32];
          tmem_ld_32x32b_x32(tm + cb * 64, v[0]);
          tmem_ld_32x32b_x32(tm + cb * 64 + 32, v[1]);
          tmem_ld_wait();
          uint8_t* box = tile + cb * 4096;
          __nv_bfloat16* dst = (which == 0 ? p.dv : p.dk) + (static_cast<long long>(kv) * p.Hk + hk) * width + cb * 64;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float* f = reinterpret_cast<const float*>(&v[i >> 2][(i & 3) * 8]);
            uint4 w = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
            if (whole) *reinterpret_cast<uint4*>(box + lane * 128 + ((i ^ (lane & 7)) << 4)) = w;
            else if (kv_ok && cb * 64 + i * 8 < width) *reinterpret_cast<uint4*>(dst + i * 8) = w;
          }
          if (whole) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (FULL) tma_store_2d(map, box, hk * width + cb * 64, row0);
              else tma_store_3d(map, box, cb * 64, hk, row0);
              bulk_commit_group();
            }
          }
        }
      }
      if (lane == 0) bulk_wait_read_all();      // shared memory may go; the grid's end waits for the rest
    }
  } else if (WITH_DQ) {
    // ---------------------------------------------------------------- dQ read-out (thread = head-dim index d)
    const int lg = warp & 3;                    // warps 10-13: TMEM lane groups 2, 3, 0, 1
    const int d = lg * 32 + lane;
    const int tid_dq = threadIdx.x - 320;       // 0..127
    float* sdq = reinterpret_cast<float*>(smem + BwdSmem::DQS);
    bool alive = true;
    if (tid_dq == 0) tma_prefetch_desc(&tmDQ);
    for (int it = 0; it < n_it; ++it) {
      const int q0 = it_q0(it);
      float v[64];
      if (alive && !mbar_wait(dq_full, it & 1, KID_ATTN_BWD, 10)) { alive = false; *s_dead_dq = 1; }
      if (alive) {
        tc_fence_after();
        tmem_ld64(tm_DQT + (static_cast<uint32_t>(lg * 32) << 16), v);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(dq_empty);
      }
      // the reduction of the previous tile has finished reading the staging tile
      if (it > 0 && tid_dq == 0) bulk_wait_read_all();
      asm volatile("bar.sync 2, 128;" ::: "memory");
      if (*s_dead_dq) break;
      // transpose: this thread's d column of the [64 q][128 d] tile (a warp writes 128 contiguous bytes per row).
      // Query rows past the end of the document carry exact zeros (their P and dS were masked), so the full tile
      // is added; rows past the end of the tensor and columns past the head are clipped by the copy engine.
#pragma unroll
      for (int col = 0; col < BW_Q; ++col) sdq[col * BW_D + d] = v[col];
      fence_proxy_async_smem();
      asm volatile("bar.sync 2, 128;" ::: "memory");
      if (tid_dq == 0) {
        if (FULL) tma_reduce_add_2d(&tmDQ, sdq, hq * BW_D, q0);
        else tma_reduce_add_3d(&tmDQ, sdq, 0, hq, q0);
        bulk_commit_group();
      }
    }
    if (tid_dq == 0) bulk_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// fp32 accumulators that a launch clears on the way
struct Cleared {
  float4* at[3];
  long long vecs[3];
};

// delta[h, t] = sum_d dO[t,h,d] * O[t,h,d].  Sixteen lanes and 16-byte loads per (t, h): 22 -> 16 us for 4096 x 32 rows.  The kernel
// reads only, so the accumulators of the kernels behind it are cleared here (71 MB in that case, 12 us as a launch of their own).
__global__ void __launch_bounds__(256)
attn_bwd_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out,
                      float* __restrict__ delta, long long T, int Hq, int Dv, const Cleared z) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < z.vecs[r]; i += static_cast<long long>(gridDim.x) * blockDim.x)
      z.at[r][i] = make_float4(0.f, 0.f, 0.f, 0.f);
  long long row = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 4;
  const int l = threadIdx.x & 15;
  const bool ok = row < T * Hq;
  if (!ok) row = T * Hq - 1;                 // both halves of a warp take part in the shuffles
  const bool in = l * 8 < Dv;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const uint4 a = in ? *reinterpret_cast<const uint4*>(dout + row * Dv + l * 8) : zero;
  const uint4 b = in ? *reinterpret_cast<const uint4*>(out + row * Dv + l * 8) : zero;
  const uint32_t as[4] = {a.x, a.y, a.z, a.w}, bs[4] = {b.x, b.y, b.z, b.w};
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 x = unpack_bf16(as[j]), y = unpack_bf16(bs[j]);
    s += x.x * y.x + x.y * y.y;
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (ok && l == 0) {
    const long long t = row / Hq;
    delta[(row - t * Hq) * T + t] = s;
  }
}

// dq (bf16) = dq_acc (fp32)
__global__ void attn_bwd_cast_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, long long n) {
  const long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  const float4 a = *reinterpret_cast<const float4*>(acc + i), b = *reinterpret_cast<const float4*>(acc + i + 4);
  uint4 w;
  w.x = pack_bf16(a.x, a.y); w.y = pack_bf16(a.z, a.w); w.z = pack_bf16(b.x, b.y); w.w = pack_bf16(b.z, b.w);
  *reinterpret_cast<uint4*>(dq + i) = w;
}

}  // namespace ttb

using namespace ttb;

template <int DQK, bool WITH_DQ, bool FULL>
static int launch_attn_bwd(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tk, const CUtensorMap& tv,
                           const CUtensorMap& tdq, const CUtensorMap& tdk, const CUtensorMap& tdv, const AttnBwdParams& p, int n_tiles,
                           cudaStream_t stream) {
  static bool smem_done[16] = {};
  using Smem = ttb::BwdSmem<DQK, WITH_DQ>;
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(attn_bwd_kernel<DQK, WITH_DQ, FULL>), Smem::TOTAL, smem_done);
  if (e != cudaSuccess) return 300 + static_cast<int>(e);
  const int heads = p.group_loop ? p.Hk : p.Hq;
  dim3 grid(WITH_DQ ? n_tiles : heads, WITH_DQ ? heads : n_tiles);
  attn_bwd_kernel<DQK, WITH_DQ, FULL><<<grid, WITH_DQ ? 448 : 320, Smem::TOTAL, stream>>>(tq, tdo, tk, tv, tdq, tdk, tdv, p);
  return 0;
}

// q: [T, Hq, D] contiguous; dout, out: [T, Hq, Dv] contiguous; k: [T, Hk, D] (ldk); v: [T, Hk, Dv] (ldv, may be strided); D and
// Dv up to 128 in multiples of 8, or D = 192 with Dv = 128.  delta fp32 [Hq*T] scratch (left filled with rowsum(dO * O) for the query-major dQ pass).
// with_dq != 0 (D <= 128 only): dQ too, reduced into dq_acc (fp32 [T*Hq*D], cleared here) and cast to dq;
// with_dq == 0: dK and dV only (dq_acc and dq unused); with_dq == 2: the same with one CTA per kv head looping over the
// query heads of its group, so that dK / dV are written once and without atomics (no accumulators needed).  dk: [T, Hk, D], dv: [T, Hk, Dv]; with Hq > Hk the fp32
// accumulators dk_acc / dv_acc (cleared here, same shapes) are required.
TTB_EXPORT int ttb_attn_bwd(const void* q, const void* k, long long ldk, const void* v, long long ldv, const void* out,
                            const void* dout, const float* lse, float* delta, float* dq_acc, float* dk_acc,
                            float* dv_acc, void* dq, void* dk, void* dv, const int* kv_tiles, int n_tiles, long long T, int Hq, int Hk, int D, int Dv, float scale,
                            int causal, int with_dq, void* stream_ptr) {
  if (D < 8 || Dv < 8 || D % 8 || Dv % 8 || Dv > BW_D || (D > 128 && !(D == 192 && Dv == BW_D)) || Hq % Hk) return 901;
  const int group_loop = with_dq == 2;
  if (group_loop) with_dq = 0;
  if (with_dq && D > 128) return 904;
  if ((ldk % 8) || (ldv % 8)) return 902;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  if (T == 0 || n_tiles == 0) return 0;
  if ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(out)) & 15) return 906;
  const bool grouped = Hq != Hk && !group_loop;
  if (with_dq && (dq_acc == nullptr || dq == nullptr)) return 905;
  if (grouped && (dk_acc == nullptr || dv_acc == nullptr)) return 903;
  const long long n[3] = {with_dq ? T * Hq * D : 0, grouped ? T * Hk * D : 0, grouped ? T * Hk * Dv : 0};
  float* acc[3] = {dq_acc, dk_acc, dv_acc};
  Cleared cleared;
  for (int i = 0; i < 3; ++i) {
    if (reinterpret_cast<uintptr_t>(acc[i]) & 15) return 906;
    cleared.at[i] = reinterpret_cast<float4*>(acc[i]);
    cleared.vecs[i] = n[i] / 4;
  }
  attn_bwd_delta_kernel<<<(unsigned)((T * Hq + 15) / 16), 256, 0, stream>>>((const __nv_bfloat16*)dout,
                                                                        (const __nv_bfloat16*)out, delta, T, Hq, Dv, cleared);
  const bool full = D >= 128 && Dv == BW_D;
  const auto map = full ? make_rows_map : make_heads_map;
  CUtensorMap tq, tdo, tk, tv;
  if (map(&tq, q, T, (long long)Hq * D, Hq, D, 64)) return 101;
  if (map(&tdo, dout, T, (long long)Hq * Dv, Hq, Dv, 64)) return 102;
  if (map(&tk, k, T, ldk, Hk, D, 128)) return 103;
  if (map(&tv, v, T, ldv, Hk, Dv, 128)) return 104;
  CUtensorMap tdq = tq;   // placeholder in the form without dQ
  if (with_dq) {
    // the staging tile's rows, clipped to the head where it is narrower
    const uint64_t dims2[2] = {static_cast<uint64_t>(Hq) * D, static_cast<uint64_t>(T)};
    const uint64_t dims3[3] = {static_cast<uint64_t>(D), static_cast<uint64_t>(Hq), static_cast<uint64_t>(T)};
    const uint64_t str[2] = {static_cast<uint64_t>(D) * 4, static_cast<uint64_t>(Hq) * D * 4};
    const uint32_t box2[2] = {static_cast<uint32_t>(BW_D), 64}, box3[3] = {static_cast<uint32_t>(BW_D), 1, 64};
    if (full ? make_tmap_f32_linear(&tdq, dq_acc, 2, dims2, str + 1, box2) : make_tmap_f32_linear(&tdq, dq_acc, 3, dims3, str, box3)) return 105;
  }
  // dK / dV: boxes of 32 rows and 128 bytes, fp32 sums or bf16 results
  CUtensorMap tdk, tdv;
  auto out_map = [&](CUtensorMap* m, float* acc, void* res, int width) {
    const int size = grouped ? 4 : 2;
    const uint64_t dims2[2] = {static_cast<uint64_t>(Hk) * width, static_cast<uint64_t>(T)};
    const uint64_t dims3[3] = {static_cast<uint64_t>(width), static_cast<uint64_t>(Hk), static_cast<uint64_t>(T)};
    const uint64_t str[2] = {static_cast<uint64_t>(width) * size, static_cast<uint64_t>(Hk) * width * size};
    const uint32_t box2[2] = {static_cast<uint32_t>(128 / size), 32}, box3[3] = {static_cast<uint32_t>(128 / size), 1, 32};
    return make_tmap_typed(m, grouped ? static_cast<const void*>(acc) : res, full ? 2 : 3, full ? dims2 : dims3, full ? str + 1 : str,
                           full ? box2 : box3, grouped ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                           CU_TENSOR_MAP_SWIZZLE_128B);
  };
  if (out_map(&tdk, dk_acc, dk, D)) return 106;
  if (out_map(&tdv, dv_acc, dv, Dv)) return 107;
  AttnBwdParams p{kv_tiles, lse, delta, dq_acc, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, dk_acc, dv_acc, Hq, Hk, D, Dv, T, scale, causal, group_loop};
  auto run = [&](auto is_full) {
    constexpr bool FULL = decltype(is_full)::value;
    return with_dq ? launch_attn_bwd<128, true, FULL>(tq, tdo, tk, tv, tdq, tdk, tdv, p, n_tiles, stream)
                   : launch_attn_bwd<128, false, FULL>(tq, tdo, tk, tv, tdq, tdk, tdv, p, n_tiles, stream);
  };
  const int rc = D == 192 ? launch_attn_bwd<192, false, true>(tq, tdo, tk, tv, tdq, tdk, tdv, p, n_tiles, stream)
                          : (full ? run(std::true_type{}) : run(std::false_type{}));
  if (rc) return rc;
  // fp32 accumulators -> bf16; the ones that lie back to back on both sides go in one launch
  __nv_bfloat16* dst[3] = {(__nv_bfloat16*)dq, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv};
  for (int i = 0; i < 3;) {
    long long run = n[i];
    int j = i + 1;
    while (j < 3 && run > 0 && acc[j] == acc[i] + run && dst[j] == dst[i] + run) run += n[j++];
    if (run > 0) attn_bwd_cast_kernel<<<(unsigned)((run / 8 + 255) / 256), 256, 0, stream>>>(acc[i], dst[i], run);
    i = j;
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}
