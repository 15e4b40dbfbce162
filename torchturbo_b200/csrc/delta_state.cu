// Chunk-state recurrence of the (gated) delta rule for sm_100a: the only sequential part of the chunked evaluation of
// GatedDeltaNet / Kimi Delta Attention layers, forward and backward.
//
// With 64-token chunks and per-chunk operands prepared by chunk-parallel (batched) GEMMs, the state S [K=128, V=128] of
// one head of one sequence obeys
//     X_c     = U_c  + s1 * A_c S            [64, V]     forward:  v_new = u - w S            (s1 = -1, A = w)
//     S      <- d_c (.) S + s2 * B_c^T X_c   [K, V]      forward:  S = d S + k_out^T v_new    (s2 = +1, B = k_out)
// and the reverse pass over the same chunks has the same shape with the operands swapped,
//     dX_c    = G_c  + k_out_c dS            (s1 = +1, A = k_out, U = gradient that reaches v_new directly)
//     dS     <- d_c (.) dS - w_c^T dX_c + GS_c   (s2 = -1, B = w, GS = gradient that reaches the chunk's start state)
// so one kernel runs both directions.  d_c is a scalar per chunk (GatedDeltaNet) or a vector over K (KDA).
//
// The columns of S do not mix, so a CTA owns 32 of the 128 value columns of one (sequence, head).  Its part of the state
// lives transposed in registers, two threads per value column v holding 64 of its 128 K-entries each in fp32 (TMEM lane = v),
// and as a bf16 K-major tile in shared memory for the tensor cores:
//     acc1 [V, 64]  = S^T  A_c^T       tcgen05, M = 128, N = 64   (K-major x K-major)
//     acc2 [V, 128] = X^T  B_c         tcgen05, M = 128, N = 128  (K-major x MN-major)
// The products keep M = 128: rows past the 32 read whatever lies behind the tile in shared memory and fill accumulator lanes that
// nobody reads (rows of a product do not mix either).
// Warp roles: 0 and 4 state warps (K-entries 0-63 and 64-127 of S), 1 and 5 x warps (tokens 0-31 and 32-63 of X), 2 loads, 3 products,
// 6 stores.  A warp reads the TMEM lanes 32 (warp % 4) .. +31, so the rows of S^T are given to the first product 32 rows down.
// The chain of a chunk is the two small products, X formed from the first and S from the second.  The 224 KB of states and rows that a
// chunk moves (all 128 columns) go through the copy engine, two chunks ahead and behind: U and the added gradient arrive in shared
// memory, X and the new state replace them there in place and leave from there.  With 64 columns a CTA and the state threads loading
// and storing their own elements a chunk was 5900 clocks forward and 12300 in reverse: stores leave an SM at 32 bytes a clock, the
// added values did not fit into registers, and the decay was waited for; with one pair of warps for X and S it was 3700 and 4300.
// CTAs stay and walk the (sequence, head, column group) items, longest sequences first: the loads of the next item overlap the end of
// the last, and a short sequence does not pay for barriers and tensor memory.
// Forward passes whose CTAs would leave a last wave partly empty take the form without any of that (`wide_pays`, below).
// Forward and reverse in us, before -> now: 32 heads, 4096 tokens in four documents (the longest 44 chunks) 140 + 252 -> 94 + 104, in
// one document 155 + 288 -> 105 + 113 (203 MB written each way, 68 at the rate of a fill), in four equal ones 70 + 117 -> 70 + 91, in 64
// of one chunk 100 + 167 -> 88 + 127; 8 heads with decay vectors, 2047 tokens 47 + 77 -> 33 + 37.
// Every wait is bounded; on a timeout the roles drain to the final barrier, TMEM is freed and the status word records
// kernel / site.
//
// Counterpart of the `chunk_gated_delta_rule` / `chunk_kda` operators that the reference takes from
// flash-linear-attention (ops/providers/native/gated_delta_rule.py, ops/providers/native/kda.py).
#include "common.cuh"

namespace ttb {

constexpr unsigned KID_DELTA_STATE = 9;
constexpr int DS_C = 64;     // tokens per chunk
constexpr int DS_D = 128;    // K = V = 128
constexpr int DS_V = 32;     // value columns per CTA
constexpr int DS_THREADS = 224;

struct DeltaStateParams {
  const float* decay;    // [H, NC] or [H, NC, 128]
  const int* seq_chunks; // [nseq, 2]: first chunk, number of chunks
  int nseq, H, NC, items;
  int vec, reverse, add;
  int first;             // state before the first chunk: 0 zero, 1 from `add` (reverse), 2 from `init`
  float s1, s2;
};

struct DsSmem {
  static constexpr int ST_PANEL = DS_V * 128;            // S^T bf16 [32 v][64 k] per panel, two panels
  static constexpr int U = 0;                            // 2 x 8 KB  U, then X: fp32 [64 c][32 v]
  static constexpr int ST = U + 2 * 8192;                // behind at least 4 KB: the first product starts 32 rows before it
  static constexpr int XT = ST + 2 * ST_PANEL;           // X^T bf16 [32 v][64 c]
  static constexpr int A = XT + DS_V * 128;              // 16 KB  A_c [64 c][128 k] (also behind the short tiles above)
  static constexpr int B = A + 16384;                    // 16 KB  B_c [64 c][128 k]
  static constexpr int G = B + 16384;                    // 2 x 16 KB  added gradient or first state, then the new state: fp32 [128 k][32 v]
  static constexpr int DEC = G + 2 * 16384;              // 2 x float [128]
  static constexpr int BARS = DEC + 2 * 512;
  static constexpr int TOTAL = BARS + 256 + 1024;
};
static_assert(2 * DsSmem::TOTAL + 2048 <= 233472, "two CTAs per SM");

__device__ __forceinline__ float ds_ld(uint32_t addr) {     // volatile: stays behind the waits
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void ds_st(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

__global__ void __launch_bounds__(DS_THREADS, 2)
delta_state_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmU,
                   const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmG, const __grid_constant__ CUtensorMap tmI,
                   const __grid_constant__ CUtensorMap tmS, const DeltaStateParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint8_t s_order[32];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + DsSmem::BARS);
  uint64_t *a_full = bars, *a_empty = bars + 1, *b_full = bars + 2, *b_empty = bars + 3;
  uint64_t *u_full = bars + 4, *u_empty = bars + 6;      // [2] U (and a decay vector) has arrived / X has left
  uint64_t *g_full = bars + 8, *g_empty = bars + 10;     // [2] the added gradient has arrived / the state has left
  uint64_t *x_done = bars + 12, *s_done = bars + 14;     // [2] X / the new state is in shared memory
  uint64_t* st_ready = bars + 16;   // S^T (bf16) of the next chunk is in shared memory
  uint64_t* acc1_full = bars + 17;
  uint64_t* x_ready = bars + 18;    // X^T (bf16) is in shared memory
  uint64_t* acc2_full = bars + 19;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slots = p.NC + p.nseq;

  if (threadIdx.x == 0) {
    mbar_init(a_full, 1); mbar_init(a_empty, 1); mbar_init(b_full, 1); mbar_init(b_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&u_full[i], 1); mbar_init(&u_empty[i], 1); mbar_init(&g_full[i], 1); mbar_init(&g_empty[i], 1);
      mbar_init(&x_done[i], 2); mbar_init(&s_done[i], 2);
    }
    mbar_init(st_ready, 2);
    mbar_init(acc1_full, 1);
    mbar_init(x_ready, 2);
    mbar_init(acc2_full, 1);
    mbar_fence_init();
  }
  if (warp == 3) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  if (warp == 1) {
    // the order of up to 32 sequences by their length, longest first
    const int mine = lane < p.nseq ? p.seq_chunks[lane * 2 + 1] : -1;
    int rank = 0;
    for (int j = 0; j < min(p.nseq, 32); ++j) {
      const int other = __shfl_sync(0xffffffffu, mine, j);
      rank += other > mine || (other == mine && j < lane);
    }
    if (lane < p.nseq) s_order[rank & 31] = static_cast<uint8_t>(lane);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tm1 = tmem_base;         // 64 columns
  const uint32_t tm2 = tmem_base + 128;   // 128 columns

  // Item: column groups of a head next to one another (they share A and B), sequences last.
  struct Item {
    int v0, h, seq, c0, n;
  };
  auto item_at = [&](int w) {
    Item x;
    const int turn = (w >> 2) / p.H;
    x.v0 = (w & 3) * DS_V;
    x.h = (w >> 2) - turn * p.H;
    x.seq = p.nseq <= 32 ? s_order[turn] : turn;
    const int2 r = __ldg(reinterpret_cast<const int2*>(p.seq_chunks) + x.seq);
    x.c0 = r.x;
    x.n = r.y;
    return x;
  };
  auto chunk_of = [&](const Item& x, int i) { return p.reverse ? x.c0 + x.n - 1 - i : x.c0 + i; };
  // row of the state behind chunk i, and of the one before the first (i = -1)
  auto state_row = [&](const Item& x, int i) {
    const int slot = (p.reverse ? x.c0 + x.n - 1 - i : x.c0 + i + 1) + x.seq;
    return (x.h * slots + slot) * DS_D;
  };
  const bool first_loaded = p.first != 0;
  const bool gated = p.add || first_loaded;           // the loading warp hands out the places of the states, with or without data in them
  // counters of this role's chunks (t) and states (g: one more per item); slot = count & 1, phase = (count >> 1) & 1
  uint32_t t = 0, g = 0;
  bool ok = true;

  if (warp == 2) {
    // ---------------------------------------------------------------- loads
    if (elect_one()) {
      tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB); tma_prefetch_desc(&tmU); tma_prefetch_desc(&tmG);
      for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
        const Item x = item_at(w);
        // the next state's place, with rows of `map` in it
        auto hand_out = [&](const CUtensorMap* map, int row) {
          const int s = g & 1;
          if (!mbar_wait(&g_empty[s], ((g >> 1) & 1) ^ 1, KID_DELTA_STATE, 9)) return false;
          if (map) {
            mbar_expect_tx(&g_full[s], 16384);
            tma_load_2d(smem + DsSmem::G + s * 16384, map, &g_full[s], x.v0, row);
          } else {
            mbar_arrive(&g_full[s]);
          }
          return true;
        };
        if (gated) {
          ok = p.first == 1 ? hand_out(&tmG, state_row(x, -1)) : hand_out(p.first ? &tmI : nullptr, (x.h * p.nseq + x.seq) * DS_D);
          if (!ok) break;
        }
        ++g;
        for (int i = 0; i < x.n; ++i, ++t, ++g) {
          const int c = chunk_of(x, i), s = t & 1, row0 = (x.h * p.NC + c) * DS_C;
          if (!(ok = mbar_wait(a_empty, (t & 1) ^ 1, KID_DELTA_STATE, 1))) break;
          mbar_expect_tx(a_full, 16384);
          tma_load_2d(smem + DsSmem::A, &tmA, a_full, 0, row0);
          tma_load_2d(smem + DsSmem::A + 8192, &tmA, a_full, 64, row0);
          if (!(ok = mbar_wait(&u_empty[s], ((t >> 1) & 1) ^ 1, KID_DELTA_STATE, 7))) break;
          mbar_expect_tx(&u_full[s], 8192 + (p.vec ? 512 : 0));
          tma_load_2d(smem + DsSmem::U + s * 8192, &tmU, &u_full[s], x.v0, row0);
          if (p.vec) bulk_load(smem + DsSmem::DEC + s * 512, p.decay + (static_cast<long long>(x.h) * p.NC + c) * DS_D, 512, &u_full[s]);
          if (!(ok = mbar_wait(b_empty, (t & 1) ^ 1, KID_DELTA_STATE, 8))) break;
          mbar_expect_tx(b_full, 16384);
          tma_load_2d(smem + DsSmem::B, &tmB, b_full, 0, row0);
          tma_load_2d(smem + DsSmem::B + 8192, &tmB, b_full, 64, row0);
          if (gated && !(ok = hand_out(p.add ? &tmG : nullptr, state_row(x, i)))) break;
        }
      }
    }
  } else if (warp == 6) {
    // ---------------------------------------------------------------- stores
    if (elect_one()) {
      tma_prefetch_desc(&tmX); tma_prefetch_desc(&tmS);
      for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
        const Item x = item_at(w);
        for (int i = -1; i < x.n; ++i, ++g) {
          const int s = g & 1;
          if (i >= 0) {
            if (!(ok = mbar_wait(&x_done[t & 1], (t >> 1) & 1, KID_DELTA_STATE, 10))) break;
            tma_store_2d(&tmX, smem + DsSmem::U + (t & 1) * 8192, x.v0, (x.h * p.NC + chunk_of(x, i)) * DS_C);
            bulk_commit_group();
          }
          if (!(ok = mbar_wait(&s_done[s], (g >> 1) & 1, KID_DELTA_STATE, 11))) break;
          tma_store_2d(&tmS, smem + DsSmem::G + s * 16384, x.v0, state_row(x, i));
          bulk_commit_group();
          bulk_wait_read_all();
          mbar_arrive(&g_empty[s]);
          if (i >= 0) {
            mbar_arrive(&u_empty[t & 1]);
            ++t;
          }
        }
      }
      bulk_wait_read_all();
    }
  } else if (warp == 3) {
    // ---------------------------------------------------------------- products (the whole warp, see umma_ss_w)
    constexpr uint32_t id1 = make_idesc_bf16(128, 64, false, false);
    constexpr uint32_t id2 = make_idesc_bf16(128, 128, false, true);
    const uint32_t leader = elect_one() ? 1u : 0u;
    const SmemDesc dST = make_smem_desc2(smem_u32(smem + DsSmem::ST) - 32 * 128, 16, 1024), dXT = make_smem_desc2(smem_u32(smem + DsSmem::XT), 16, 1024);
    const SmemDesc dA = make_smem_desc2(smem_u32(smem + DsSmem::A), 16, 1024), dB = make_smem_desc2(smem_u32(smem + DsSmem::B), 8192, 1024);
    for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
      const Item x = item_at(w);
      for (int i = 0; i < x.n; ++i, ++t) {
        if (!(ok = mbar_wait(a_full, t & 1, KID_DELTA_STATE, 2))) break;
        if (!(ok = mbar_wait(st_ready, t & 1, KID_DELTA_STATE, 3))) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)      // reduction over k = 128
          umma_ss_w(leader, tm1, desc_at(dST, (kk >> 2) * DsSmem::ST_PANEL + (kk & 3) * 32), desc_at(dA, (kk >> 2) * 8192 + (kk & 3) * 32), id1, kk != 0);
        umma_commit_w(leader, acc1_full);
        umma_commit_w(leader, a_empty);
        if (!(ok = mbar_wait(b_full, t & 1, KID_DELTA_STATE, 12))) break;
        if (!(ok = mbar_wait(x_ready, t & 1, KID_DELTA_STATE, 4))) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)      // reduction over the 64 tokens of the chunk
          umma_ss_w(leader, tm2, desc_at(dXT, kk * 32), desc_at(dB, kk * 2048), id2, kk != 0);
        umma_commit_w(leader, acc2_full);
        umma_commit_w(leader, b_empty);
      }
    }
  } else {
    const int half = warp >> 2;                  // of the K-entries / tokens
    auto signal = [&](uint64_t* bar) {           // what this warp has written to shared memory is there for the async proxy
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    if (warp & 1) {
      // ---------------------------------------------------------------- x warps (two threads per value column, TMEM lanes 32-63)
      const uint32_t lanes = 32u << 16, sXT = smem_u32(smem + DsSmem::XT) + lane * 128;
      for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
        const Item x = item_at(w);
        for (int i = 0; i < x.n; ++i, ++t) {
          const int s = t & 1;
          const uint32_t sU = smem_u32(smem + DsSmem::U) + s * 8192 + (half * 32 * DS_V + lane) * 4;
          if (!(ok = mbar_wait(&u_full[s], (t >> 1) & 1, KID_DELTA_STATE, 13))) break;
          float u[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) u[j] = ds_ld(sU + j * DS_V * 4);
          if (!(ok = mbar_wait(acc1_full, t & 1, KID_DELTA_STATE, 5))) break;
          tc_fence_after();
          uint32_t r[32];
          tmem_ld_32x32b_x32(tm1 + half * 32 + lanes, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) u[j] = fmaf(p.s1, __uint_as_float(r[j]), u[j]);
#pragma unroll
          for (int ch = 0; ch < 4; ++ch)
            st_shared_v4(sXT + (((half * 4 + ch) ^ (lane & 7)) * 16), pack_bf16(p.s2 * u[ch * 8 + 0], p.s2 * u[ch * 8 + 1]),
                         pack_bf16(p.s2 * u[ch * 8 + 2], p.s2 * u[ch * 8 + 3]), pack_bf16(p.s2 * u[ch * 8 + 4], p.s2 * u[ch * 8 + 5]),
                         pack_bf16(p.s2 * u[ch * 8 + 6], p.s2 * u[ch * 8 + 7]));
          tc_fence_before();
          signal(x_ready);
#pragma unroll
          for (int j = 0; j < 32; ++j) ds_st(sU + j * DS_V * 4, u[j]);
          signal(&x_done[s]);
        }
      }
    } else {
      // ---------------------------------------------------------------- state warps (two threads per value column, TMEM lanes 0-31)
      float S[64];
      const uint32_t sST = smem_u32(smem + DsSmem::ST) + half * DsSmem::ST_PANEL + lane * 128;
      // this half of row v of S^T -> bf16 K-major panel (128-byte swizzle)
      auto publish = [&]() {
#pragma unroll
        for (int ch = 0; ch < 8; ++ch)
          st_shared_v4(sST + ((ch ^ (lane & 7)) * 16), pack_bf16(S[ch * 8 + 0], S[ch * 8 + 1]), pack_bf16(S[ch * 8 + 2], S[ch * 8 + 3]),
                       pack_bf16(S[ch * 8 + 4], S[ch * 8 + 5]), pack_bf16(S[ch * 8 + 6], S[ch * 8 + 7]));
        signal(st_ready);
      };
      const uint32_t sG0 = smem_u32(smem + DsSmem::G) + (half * 64 * DS_V + lane) * 4;
      for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
        const Item x = item_at(w);
        // a chunk's own decay, asked for a chunk ahead (volatile: the compiler would move a plain load down to its use)
        auto decay_of = [&](int i) {
          float d;
          asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(d) : "l"(p.decay + static_cast<long long>(x.h) * p.NC + chunk_of(x, i)));
          return d;
        };
        float dec_next = !p.vec && x.n > 0 ? decay_of(0) : 1.f;
        // the state before the first chunk, which its slot records too
        {
          const int s = g & 1;
          const uint32_t ph = (g >> 1) & 1, sG = sG0 + s * 16384;
          if (!(ok = gated ? mbar_wait(&g_full[s], ph, KID_DELTA_STATE, 14) : mbar_wait(&g_empty[s], ph ^ 1, KID_DELTA_STATE, 15))) break;
          if (first_loaded) {
#pragma unroll
            for (int k = 0; k < 64; ++k) S[k] = ds_ld(sG + k * DS_V * 4);
          } else {
#pragma unroll
            for (int k = 0; k < 64; ++k) { S[k] = 0.f; ds_st(sG + k * DS_V * 4, 0.f); }
          }
          if (x.n > 0) publish();
          signal(&s_done[s]);
          ++g;
        }
        for (int i = 0; i < x.n; ++i, ++t, ++g) {
          const int s = g & 1;
          const uint32_t ph = (g >> 1) & 1, sG = sG0 + s * 16384, sD = smem_u32(smem + DsSmem::DEC) + (t & 1) * 512 + half * 256;
          const float dec = dec_next;
          if (!p.vec && i + 1 < x.n) dec_next = decay_of(i + 1);
          // the added gradient is there, or the state of two steps ago has left its place; a decay vector came with U
          if (!(ok = gated ? mbar_wait(&g_full[s], ph, KID_DELTA_STATE, 14) : mbar_wait(&g_empty[s], ph ^ 1, KID_DELTA_STATE, 15))) break;
          if (p.vec && !(ok = mbar_wait(&u_full[t & 1], (t >> 1) & 1, KID_DELTA_STATE, 16))) break;
          if (!(ok = mbar_wait(acc2_full, t & 1, KID_DELTA_STATE, 6))) break;
          tc_fence_after();
#pragma unroll
          for (int cb = 0; cb < 2; ++cb) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(tm2 + half * 64 + cb * 32, r);
            tmem_ld_wait();
            if (p.vec) {
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                uint32_t d[4];
                ld_shared_v4(sD + (cb * 32 + j) * 4, d[0], d[1], d[2], d[3]);
#pragma unroll
                for (int e = 0; e < 4; ++e) S[cb * 32 + j + e] = fmaf(__uint_as_float(d[e]), S[cb * 32 + j + e], __uint_as_float(r[j + e]));
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) S[cb * 32 + j] = fmaf(dec, S[cb * 32 + j], __uint_as_float(r[j]));
            }
            if (p.add) {
#pragma unroll
              for (int j = 0; j < 32; ++j) S[cb * 32 + j] += ds_ld(sG + (cb * 32 + j) * DS_V * 4);
            }
          }
          tc_fence_before();
          if (i + 1 < x.n) publish();
#pragma unroll
          for (int k = 0; k < 64; ++k) ds_st(sG + k * DS_V * 4, S[k]);
          signal(&s_done[s]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// Forward pass in CTAs of 64 columns whose threads load U and store X and the states themselves: warps 0, 1, 4, 5 hold the state and form X
// (warps 4 and 5 K-entries 64-127 and tokens 32-63), 2 loads the operands (two stages), 3 issues the products.
struct DsWideParams {
  const float *U, *decay, *init;
  float *X, *states;
  const int* seq_chunks;
  int nseq, NC, vec;
  float s1, s2;
};

struct DsWideSmem {
  static constexpr int V = 64;                           // value columns
  static constexpr int ST_PANEL = V * 128;               // S^T bf16 [64 v][64 k] per panel, two panels
  static constexpr int ST = 0;
  static constexpr int XT = ST + 2 * ST_PANEL;           // X^T bf16 [64 v][64 c]
  static constexpr int A = XT + V * 128;                 // 2 x 16 KB  A_c [64 c][128 k] (also behind the short tiles above)
  static constexpr int B = A + 2 * 16384;                // 2 x 16 KB  B_c [64 c][128 k]
  static constexpr int DEC = B + 2 * 16384;              // float [128]
  static constexpr int BARS = DEC + 512;
  static constexpr int TOTAL = BARS + 256 + 1024;
};

__global__ void __launch_bounds__(192, 2)
delta_state_wide_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const DsWideParams p) {
  using L = DsWideSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t *ab_full = bars, *ab_empty = bars + 2;        // [2]
  uint64_t *st_ready = bars + 4, *acc1_full = bars + 5, *x_ready = bars + 6, *acc2_full = bars + 7;      // as above
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  volatile int* s_dead = reinterpret_cast<volatile int*>(bars + 9);      // a state warp's wait gave up
  float* s_dec = reinterpret_cast<float*>(smem + L::DEC);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seq = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * L::V, slots = p.NC + p.nseq;
  const int c0 = p.seq_chunks[seq * 2], n = p.seq_chunks[seq * 2 + 1];

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&ab_full[i], 1); mbar_init(&ab_empty[i], 1); }
    mbar_init(st_ready, 4); mbar_init(acc1_full, 1); mbar_init(x_ready, 4); mbar_init(acc2_full, 1);
    *s_dead = 0;
    mbar_fence_init();
  }
  if (warp == 3) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot, tm1 = tmem_base, tm2 = tmem_base + 128;

  if (warp == 2) {
    if (elect_one()) {
      tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB);
      for (int i = 0; i < n; ++i) {
        const int st = i & 1, row0 = (h * p.NC + c0 + i) * DS_C;
        if (!mbar_wait(&ab_empty[st], ((i >> 1) & 1) ^ 1, KID_DELTA_STATE, 17)) break;
        mbar_expect_tx(&ab_full[st], 32768);
        uint8_t *sa = smem + L::A + st * 16384, *sb = smem + L::B + st * 16384;
        tma_load_2d(sa, &tmA, &ab_full[st], 0, row0);
        tma_load_2d(sa + 8192, &tmA, &ab_full[st], 64, row0);
        tma_load_2d(sb, &tmB, &ab_full[st], 0, row0);
        tma_load_2d(sb + 8192, &tmB, &ab_full[st], 64, row0);
      }
    }
  } else if (warp == 3) {
    constexpr uint32_t id1 = make_idesc_bf16(128, 64, false, false), id2 = make_idesc_bf16(128, 128, false, true);
    if (elect_one()) {
      const uint32_t sST = smem_u32(smem + L::ST), sXT = smem_u32(smem + L::XT);
      for (int i = 0; i < n; ++i) {
        const int st = i & 1;
        if (!mbar_wait(&ab_full[st], (i >> 1) & 1, KID_DELTA_STATE, 18)) break;
        if (!mbar_wait(st_ready, i & 1, KID_DELTA_STATE, 19)) break;
        tc_fence_after();
        const uint32_t sA = smem_u32(smem + L::A + st * 16384), sB = smem_u32(smem + L::B + st * 16384);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)    // reduction over k = 128
          umma_ss(tm1, make_smem_desc(sST + (kk >> 2) * L::ST_PANEL + (kk & 3) * 32, 16, 1024),
                  make_smem_desc(sA + (kk >> 2) * 8192 + (kk & 3) * 32, 16, 1024), id1, kk != 0);
        umma_commit(acc1_full);
        if (!mbar_wait(x_ready, i & 1, KID_DELTA_STATE, 20)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)    // reduction over the 64 tokens of the chunk
          umma_ss(tm2, make_smem_desc(sXT + kk * 32, 16, 1024), make_smem_desc(sB + kk * 2048, 8192, 1024), id2, kk != 0);
        umma_commit(acc2_full);
        umma_commit(&ab_empty[st]);
      }
    }
  } else {
    const int half = warp >> 2, vl = (warp & 3) * 32 + lane, v = v0 + vl, k0 = half * 64, t0 = half * 32;   // this thread's column, K-entries, tokens
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    uint8_t *sST = smem + L::ST + half * L::ST_PANEL + vl * 128, *sXT = smem + L::XT + vl * 128;
    float S[64], u[32];
    auto state_at = [&](int slot) { return p.states + ((static_cast<long long>(h) * slots + slot) * DS_D + k0) * DS_D + v; };
    auto row_at = [&](int i) { return ((static_cast<long long>(h) * p.NC + c0 + i) * DS_C + t0) * DS_D + v; };
    auto signal = [&](uint64_t* bar) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto publish = [&]() {
#pragma unroll
      for (int ch = 0; ch < 8; ++ch)
        *reinterpret_cast<uint4*>(sST + ((ch ^ (lane & 7)) * 16)) = make_uint4(pack_bf16(S[ch * 8 + 0], S[ch * 8 + 1]), pack_bf16(S[ch * 8 + 2], S[ch * 8 + 3]),
                                                                               pack_bf16(S[ch * 8 + 4], S[ch * 8 + 5]), pack_bf16(S[ch * 8 + 6], S[ch * 8 + 7]));
      signal(st_ready);
    };
    auto fetch_u = [&](int i) {
      const float* src = p.U + row_at(i);
#pragma unroll
      for (int j = 0; j < 32; ++j) u[j] = __ldg(src + j * DS_D);
    };
    {
      const float* src = p.init ? p.init + ((static_cast<long long>(h) * p.nseq + seq) * DS_D + k0) * DS_D + v : nullptr;
      float* dst = state_at(c0 + seq);
#pragma unroll
      for (int k = 0; k < 64; ++k) S[k] = src ? __ldg(src + k * DS_D) : 0.f;
#pragma unroll
      for (int k = 0; k < 64; ++k) dst[k * DS_D] = S[k];
    }
    if (n > 0) {
      publish();
      fetch_u(0);
    }
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      // the decay is asked for ahead of the first wait: a load behind the second one would be on the chain
      const long long chunk = static_cast<long long>(h) * p.NC + c0 + i;
      const float dec = __ldg(p.decay + (p.vec ? chunk * DS_D + half * L::V + vl : chunk));
      if (ok && mbar_wait(acc1_full, i & 1, KID_DELTA_STATE, 21)) {
        tc_fence_after();
        uint32_t r[32];
        tmem_ld_32x32b_x32(tm1 + t0 + lanes, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) u[j] = fmaf(p.s1, __uint_as_float(r[j]), u[j]);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
          *reinterpret_cast<uint4*>(sXT + (((half * 4 + ch) ^ (lane & 7)) * 16)) =
              make_uint4(pack_bf16(p.s2 * u[ch * 8 + 0], p.s2 * u[ch * 8 + 1]), pack_bf16(p.s2 * u[ch * 8 + 2], p.s2 * u[ch * 8 + 3]),
                         pack_bf16(p.s2 * u[ch * 8 + 4], p.s2 * u[ch * 8 + 5]), pack_bf16(p.s2 * u[ch * 8 + 6], p.s2 * u[ch * 8 + 7]));
        tc_fence_before();
        signal(x_ready);
        // off the chain, while the second product runs: X goes out, the next U comes in, and a decay vector is staged for all threads (its
        // last readers have published the state that this chunk's first product waited for)
        float* xout = p.X + row_at(i);
#pragma unroll
        for (int j = 0; j < 32; ++j) xout[j * DS_D] = u[j];
        if (i + 1 < n) fetch_u(i + 1);
        if (p.vec) s_dec[half * L::V + vl] = dec;
      } else {
        *s_dead = 1;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");     // the decay vector is staged; a failed wait is published
      if (*s_dead) break;
      if (!mbar_wait(acc2_full, i & 1, KID_DELTA_STATE, 22)) {
        ok = false;
        continue;                                        // to the barrier of the next chunk, which the other warps wait at
      }
      tc_fence_after();
#pragma unroll
      for (int cb = 0; cb < 2; ++cb) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tm2 + k0 + cb * 32 + lanes, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int k = cb * 32 + j;
          S[k] = fmaf(p.vec ? s_dec[k0 + k] : dec, S[k], __uint_as_float(r[j]));
        }
      }
      tc_fence_before();
      if (i + 1 < n) publish();
      float* dst = state_at(c0 + i + 1 + seq);
#pragma unroll
      for (int k = 0; k < 64; ++k) dst[k * DS_D] = S[k];
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// Whether a forward pass takes the form with 64 columns a CTA (the same bits).  It moves less through shared memory per column, so that two
// of its CTAs hold an SM up less, but its chain is longer (2.3 us a chunk alone on an SM, 1.5 with 32 columns).  `places` CTAs of either
// form run at once; the lines are those of sequence-and-head pairs at 148 SMs, times in us for 32 and for 64 columns:
//  * 75 to 148 pairs: all of its CTAs run at once, where a last wave of the other form's is partly empty, if no sequence is much
//    longer than the others (those of the last wave are the shortest): 32 heads with four of 16 chunks 78 and 70, of 24 110 and 100, with
//    three of 21 88 and 81.  Lengths with a mean of 0.83 of the longest 92 and 88, of 0.71 115 and 123; 80 pairs at 0.80 76 and 78, 96 at 0.88
//    82 and 84, whose shorter last wave is less of a loss;
//  * 223 to 259: two full waves against three and a bit: 240 pairs of 24 chunks 203 and 195, 256 205 and 203, 288 219 and 231; with a mean of
//    0.89 of the longest 224 170 and 168, but 256 170 and 176;
//  * sequences of one chunk, which have no chain: 64 pairs 12.3 and 10.2, 128 14.3 and 12.3, 256 20.5 and 18.4; 512 29.7 and 30.7, with first
//    states 35.8 and 38.9.
// Outside these it is 1.0 to 1.5 times slower (1 pair to 74: 1.4; 160 to 192: 1.1; 320: 1.1).
static bool wide_pays(int nseq, int H, int NC, int longest, long long places) {
  const long long pairs = static_cast<long long>(nseq) * H;
  if (longest <= 0 || H > 65535) return false;
  if (longest == 1) return pairs <= places;
  const long long mean = 20ll * NC, top = static_cast<long long>(longest) * nseq;      // of the lengths, in twentieths, and the longest
  if (2 * pairs <= places) return 4 * pairs > places && mean >= (8 * pairs < 3 * places ? 18 : 16) * top;
  return 4 * pairs > 3 * places && 8 * pairs <= 7 * places && mean >= 19 * top;
}

}  // namespace ttb

using namespace ttb;

// A, B: bf16 [H * NC * 64, 128] (chunk-major rows); U, X: fp32 [H, NC, 64, 128]; decay fp32 [H, NC] or [H, NC, 128];
// init fp32 [H, nseq, 128, 128] or null; add, states fp32 [H, NC + nseq, 128, 128] (add may be null when forward).  reverse: 0, 1, or
// 2 for a first state of zero, whose slot of `add` is then not read.  longest: chunks of the longest sequence (0: not known).
TTB_EXPORT int ttb_delta_state_scan(const void* A, const void* B, const float* U, float* X, const float* decay, int vec,
                                    const float* init, const float* add, float* states, const int* seq_chunks, int nseq,
                                    int H, int NC, int longest, int reverse, float s1, float s2, void* stream_ptr) {
  if (nseq <= 0 || H <= 0 || NC <= 0) return 0;
  if (reverse && add == nullptr) return 911;
  const long long items = static_cast<long long>(DS_D / DS_V) * H * nseq;
  if (items > 0x3fffffff) return 912;
  if ((vec && (reinterpret_cast<uintptr_t>(decay) & 15)) || (reinterpret_cast<uintptr_t>(seq_chunks) & 7)) return 913;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  CUtensorMap ta, tb, tu, tx, tg, ti, ts;
  const uint64_t rows = static_cast<uint64_t>(H) * NC * DS_C, srows = static_cast<uint64_t>(H) * (NC + nseq) * DS_D;
  {
    const uint64_t dims[2] = {DS_D, rows}, sdims[2] = {DS_D, srows}, idims[2] = {DS_D, static_cast<uint64_t>(H) * nseq * DS_D};
    const uint64_t str[1] = {DS_D * 2}, fstr[1] = {DS_D * 4};
    const uint32_t box[2] = {64, 64}, ubox[2] = {DS_V, DS_C}, sbox[2] = {DS_V, DS_D};
    if (make_tmap_bf16(&ta, A, 2, dims, str, box)) return 101;
    if (make_tmap_bf16(&tb, B, 2, dims, str, box)) return 102;
    if (make_tmap_f32_linear(&tu, U, 2, dims, fstr, ubox)) return 103;
    if (make_tmap_f32_linear(&tx, X, 2, dims, fstr, ubox)) return 104;
    if (make_tmap_f32_linear(&ts, states, 2, sdims, fstr, sbox)) return 105;
    tg = ti = ts;         // placeholders
    if (add && make_tmap_f32_linear(&tg, add, 2, sdims, fstr, sbox)) return 106;
    if (init && !reverse && make_tmap_f32_linear(&ti, init, 2, idims, fstr, sbox)) return 107;
  }
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 301;
  if (!reverse && add == nullptr && wide_pays(nseq, H, NC, longest, 2ll * sms)) {
    const DsWideParams w{U, decay, init, X, states, seq_chunks, nseq, NC, vec, s1, s2};
    static bool wide_done[16] = {};
    const cudaError_t es = ensure_dynamic_smem(reinterpret_cast<const void*>(delta_state_wide_kernel), DsWideSmem::TOTAL, wide_done);
    if (es != cudaSuccess) return 300 + static_cast<int>(es);
    delta_state_wide_kernel<<<dim3(nseq, H, DS_D / DsWideSmem::V), 192, DsWideSmem::TOTAL, stream>>>(ta, tb, w);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : 400 + (int)e;
  }
  DeltaStateParams p{decay, seq_chunks, nseq, H, NC, static_cast<int>(items), vec, reverse != 0, add != nullptr,
                     reverse == 1 ? 1 : !reverse && init ? 2 : 0, s1, s2};
  static bool done[16] = {};
  const cudaError_t es = ensure_dynamic_smem(reinterpret_cast<const void*>(delta_state_kernel), DsSmem::TOTAL, done);
  if (es != cudaSuccess) return 300 + static_cast<int>(es);
  const unsigned grid = static_cast<unsigned>(items < 2ll * sms ? items : 2ll * sms);
  delta_state_kernel<<<grid, DS_THREADS, DsSmem::TOTAL, stream>>>(ta, tb, tu, tx, tg, ti, ts, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}
