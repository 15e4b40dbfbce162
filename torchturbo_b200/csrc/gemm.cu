// Persistent, warp-specialised bf16 GEMM for sm_100a: TMA -> shared (128B swizzle)
// -> tcgen05.mma (M=128, or M=256 by a pair of CTAs, see `pays_in_pairs`) -> TMEM (double-buffered accumulator)
// -> tcgen05.ld epilogue.  One kernel body covers
//   * dense  C[M,N] = A . B          with A / B each K-major or MN-major in memory,
//   * grouped-M (MoE forward / dX): rows are grouped by expert in 128-row aligned
//     segments, `tile_group[m_tile]` names the expert whose B[g] the tile uses
//     (-1 skips the tile).  Offsets live on the device; the host never syncs.
//   * grouped-K (MoE dW): C[g] = A[rows_g]^T . B[rows_g] with row ranges from a
//     device array (64-aligned, pad rows are zero).
// Epilogues: plain store (bf16 or fp32, optional accumulate / residual add) and
// SwiGLU (gate and up column panels are loaded side by side into one 256-wide
// accumulator; out = silu(g) * u * row_scale, pre-activations optionally kept).
//
//
// Expert-parallel fusion (grouped-M only, both optional, see `EpFuse`):
//   * push prologue: two extra warps per CTA copy this rank's routed token rows (plus routing weight and a
//     return tag) straight into the owning ranks' expert-major receive buffers over NVLink while the tensor
//     cores work; rows travel in (local expert, owner) order and every (source, expert) pair raises a flag on
//     the owner when its last row has landed.  The TMA producer warp waits (bounded) for the flags of a
//     tile's expert the first time the CTA meets it, so the math of the first experts overlaps the transfer
//     of the later ones.  This is the token dispatch all-to-all of the reference
//     (models/modules/moe/token_dispatcher.py:149-201) inside the fc1 GEMM.
//   * scatter epilogue: every output row is stored straight into the source rank's [T*k, N] return buffer at
//     the position its tag names (peer stores from the epilogue warps); the last CTA raises a "rows
//     returned" flag on every peer.  This is the combine all-to-all (token_dispatcher.py:203-236) inside the
//     fc2 / input-gradient GEMM.
//
// Replaces cuBLAS `F.linear`, `grouped_gemm.ops.gmm` and the torch.compile'd
// SwiGLU of the reference (ops/providers/cuda/grouped_matmul.py:19-36,
// ops/providers/cuda/swiglu.py:26-36, models/modules/moe/experts.py:181-254).
#include "peer.cuh"
#include <cstring>

namespace ttb {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr unsigned KID_GEMM = 1;

enum Epi : int { EPI_STORE = 0, EPI_SWIGLU = 1 };

// Expert-parallel fusion parameters (device side).
struct EpFuse {
  PeerTable peers;
  // push prologue
  int push_on;
  long long off_rows, off_vals, off_tags, off_flags;  // byte offsets inside every rank's symmetric buffer
  const __nv_bfloat16* src;   // [T, lds] local token rows
  long long lds;
  const int* order;           // [n_entries] entry ids (token * k + slot) in send order
  const int* expert;          // [n_entries] global expert of every entry
  const int* dest_row;        // [n_entries] row on the owner
  const float* val;           // [n_entries] scalar that travels with the row, or null
  const int* counts;          // [E] rows this rank sends per global expert
  int* sent;                  // [E + 1] rows sent per expert, then the next chunk to claim; all zero at launch
  int n_entries, k, H, El, W, rank, epoch;
  long long cap_rows;
  unsigned long long budget_ns;
  int* status;
  // scatter epilogue
  int scat_on;
  long long off_ret, off_ret_vals, off_ret_flags;
  const int* row_tag;         // [M] tags of this rank's received rows
  const float* row_val;       // [M] scalar returned with the row, or null
  int ret_epoch;
  unsigned int* done_counter;
  int ret_rows;               // rows of every rank's return buffer (tags at or past it are refused)
};

// n / d for 0 <= n < 2^31 by a multiplication: with 2^s >= d and m = ceil(2^(31 + s) / d), m d exceeds 2^(31 + s) by less than 2^s, so
// that n m / 2^(31 + s) stays below the next whole number.
struct FastDiv {
  uint32_t mul, shift;
  __device__ __forceinline__ int operator()(int n) const { return static_cast<int>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * mul) >> shift); }
};
static FastDiv fast_div(int d) {
  uint32_t s = 0;
  while ((1ull << s) < static_cast<uint64_t>(d)) ++s;
  return FastDiv{static_cast<uint32_t>(((1ull << (31 + s)) + d - 1) / d), 31 + s};
}

struct GemmParams {
  EpFuse ep;
  int M, N, K;   // per-problem extents (N = output columns; for SwiGLU N = F)
  int m_tiles, n_tiles, groups_k;  // groups_k > 0 => grouped-K problem count
  void* C;
  long long ldc;         // elements
  long long c_group_stride;  // elements between C[g] (grouped-K)
  int c_fp32;            // 1: fp32 output, 0: bf16
  int accumulate;        // C += result (read-modify-write)
  const __nv_bfloat16* residual;  // optional [M, ldr] added before store (bf16 out)
  long long ldr;
  const int* tile_group;  // grouped-M: [m_tiles]
  const int* group_rows;  // grouped-K: [groups_k + 1], multiples of BK
  // SwiGLU
  int F;                  // gate columns [0,F), up columns [F,2F)
  const float* row_scale; // optional [M]
  __nv_bfloat16* preact;  // optional [M, ld_preact] receives gate|up
  long long ld_preact;
  const float* alpha;     // optional device scalar multiplied into the product (plain stores)
  int tma_out;            // plain bf16 rows: stored by the copy engine through the map of C
  FastDiv by_group, by_band, by_rest;   // tile counts: of a group, of a whole band, rows of the last band
  int k_splits, kb_per_split;  // > 1: "group" g covers k-blocks [g, g + 1) * kb_per_split of one product, stored at C[g]
};

template <int BN, bool PAIR>
struct SmemLayout {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * BK * 2;   // a CTA of a pair holds half of the tile's columns
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (BN == 256 && !PAIR) ? 4 : 6;
  static constexpr int EPI_STAGE_BYTES = 32 * 32 * 4;   // one 32-row x 32-column fp32 chunk per epilogue warp
  static constexpr int EPI_BYTES = 8 * EPI_STAGE_BYTES;
  static constexpr int TOTAL = STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};

constexpr int EPI_WARPS = 8;                       // two warps per TMEM lane quarter, each takes half of the columns
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;
constexpr int PUSH_WARPS = 2;                      // extra warps of a launch with the push prologue
constexpr int GEMM_THREADS_PUSH = GEMM_THREADS + 32 * PUSH_WARPS;
constexpr int PUSH_CHUNK = 8;                      // rows a push warp copies between two system-scope fences
static_assert(EPI_WARPS == 8, "the staging area is sized for eight epilogue warps");

// Epilogue staging.  tcgen05.ld hands every lane 32 consecutive columns of ITS row, so direct stores touch 32 rows per
// instruction with 16 bytes each.  The chunk is instead parked in shared memory (fp32, 128 bytes per row, 16-byte
// pieces XOR-swizzled by the row so that neither side has more than the unavoidable 4-way bank split) and written
// out row-major: one instruction stores whole 64-byte (bf16) or 128-byte (fp32) row segments of 8 or 4 rows.
__device__ __forceinline__ uint32_t epi_piece_addr(uint32_t base, int row, int piece) {
  return base + row * 128 + ((piece ^ (row & 7)) << 4);
}
// same for packed bf16 chunks: 64 bytes per row, four 16-byte pieces
__device__ __forceinline__ uint32_t epi_piece_addr64(uint32_t base, int row, int piece) {
  return base + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4);
}

template <int BN, bool A_MN, bool B_MN, int EPI, bool PAIR>
__global__ void __launch_bounds__(GEMM_THREADS_PUSH, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
            const GemmParams p) {
  using L = SmemLayout<BN, PAIR>;
  constexpr int STAGES = L::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi_stage = smem + STAGES * L::STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * L::STAGE_BYTES + L::EPI_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = bars + 2 * STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);

  __shared__ uint32_t s_landed[32];   // push prologue: experts (up to 1024) whose rows are known to have landed
  __shared__ int s_last_cta;
  __shared__ int s_dead;              // the exchange this launch belongs to has already failed: no tile is computed

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = PAIR ? static_cast<int>(cluster_ctarank()) : 0;   // CTA of the pair
  // tiles are walked by CTAs, or by pairs of them
  const int walker = PAIR ? blockIdx.x >> 1 : blockIdx.x, walkers = PAIR ? gridDim.x >> 1 : gridDim.x;
  // With the push prologue the producer may spend up to the exchange budget waiting for a peer's rows; the warps
  // downstream of it (MMA issuer, epilogue) must outwait it, or they give up on tiles whose rows arrive later.
  const uint64_t consumer_budget = p.ep.push_on ? p.ep.budget_ns + kWaitBudgetNs : kWaitBudgetNs;

  if (threadIdx.x < 32) s_landed[threadIdx.x] = 0u;
  if (threadIdx.x == 0) {
    // rows of a failed exchange never arrive: without this every CTA would sit out the full wait budget per launch
    s_dead = (p.ep.status != nullptr && *reinterpret_cast<volatile int*>(p.ep.status) != 0) ? 1 : 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], PAIR ? 2 * EPI_WARPS : EPI_WARPS);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(tmem_slot, 2 * BN);
    } else {
      tmem_alloc(tmem_slot, 2 * BN);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();     // the barriers of both CTAs are set up
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int groups = p.groups_k > 0 ? p.groups_k : p.k_splits;
  const int tiles_per_group = p.m_tiles * p.n_tiles;      // the launch checks that all tiles can be counted in 31 bits
  const int total_tiles = s_dead ? 0 : tiles_per_group * groups;

  // Decode tile -> (g, m_tile, n_tile).  Tiles are walked in bands of RASTER_M m-tiles: inside a band m runs
  // fastest, then n, so the ~148 tiles in flight cover a near-square RASTER_M x (148 / RASTER_M) block of C.  Per wave
  // that needs RASTER_M A panels and ~9 B panels instead of every A panel, and a band's A panels stay in L2 while
  // its n-tiles are walked (an m-fastest walk over all m-tiles re-read A from DRAM once per n-tile column).
  // A pair's tile has 256 rows, so its bands have half as many; `mt` is the 128-row tile of this CTA.
  constexpr int RASTER_M = PAIR ? 8 : 16;
  // What a tile reads from memory (its expert, or the row range of its group) is asked for a tile ahead: a tile of a grouped weight
  // gradient at 256 rows an expert is 2600 clocks of products, and the load in front of them was 400 to 800.
  struct Tile {
    int g, mt, nt;    // mt: 128-row tile of this CTA
    int a, b;         // grouped-M: a = expert; grouped-K: row range
  };
  auto fetch = [&](int t) {
    Tile x{0, 0, 0, 0, 0};
    if (t >= total_tiles) return x;
    x.g = p.by_group(t);
    const int r = t - x.g * tiles_per_group;
    const int band = p.by_band(r);
    const int m_base = band * RASTER_M;
    const int w = r - band * RASTER_M * p.n_tiles;
    const int left = p.m_tiles - m_base;
    x.nt = left < RASTER_M ? p.by_rest(w) : w / RASTER_M;
    x.mt = m_base + w - x.nt * (left < RASTER_M ? left : RASTER_M);
    if (PAIR) x.mt = 2 * x.mt + rank;
    if (p.tile_group) {
      x.a = __ldg(p.tile_group + x.mt);
    } else if (p.groups_k > 0) {
      x.a = __ldg(p.group_rows + x.g);
      x.b = __ldg(p.group_rows + x.g + 1);
    }
    return x;
  };
  auto unused = [&](const Tile& x) { return p.tile_group != nullptr && x.a < 0; };
  // k-range of a tile: dense -> [0, K); split -> its share of [0, K); grouped-K -> rows of group g.
  auto krange = [&](const Tile& x, int& k0, int& nkb) {
    if (p.groups_k > 0) {
      k0 = x.a;
      nkb = (x.b - x.a) / BK;
    } else if (p.k_splits > 1) {
      const int kb0 = x.g * p.kb_per_split;
      k0 = kb0 * BK;
      nkb = min(p.kb_per_split, (p.K + BK - 1) / BK - kb0);
    } else {
      k0 = 0;
      nkb = (p.K + BK - 1) / BK;
    }
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    int stage = 0;
    uint32_t phase = 0;
    // all k-blocks of one tile; run by one thread
    auto load_tile = [&](const Tile& x) -> bool {
      int k0, nkb;
      krange(x, k0, nkb);
      const int m0 = x.mt * BM;
      const int n0 = x.nt * (EPI == EPI_SWIGLU ? BN / 2 : BN);
      const int bgroup = p.tile_group ? x.a : 0;
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, KID_GEMM, 1)) return false;
        uint8_t* sa = smem + stage * L::STAGE_BYTES;
        uint8_t* sb = sa + L::A_BYTES;
        // a pair's loads all complete on the leading CTA's barrier, which expects both shares
        const uint32_t bar = PAIR ? leader_addr(&full[stage]) : 0u;
        if (rank == 0) mbar_expect_tx(&full[stage], (PAIR ? 2 : 1) * L::STAGE_BYTES);
        auto load_a = [&](void* dst, int x, int y) {
          if (PAIR) tma_load_2d_pair(dst, &tmA, bar, x, y);
          else tma_load_2d(dst, &tmA, &full[stage], x, y);
        };
        auto load_b = [&](void* dst, int x, int y) {
          if (PAIR) tma_load_3d_pair(dst, &tmB, bar, x, y, bgroup);
          else tma_load_3d(dst, &tmB, &full[stage], x, y, bgroup);
        };
        const int kc = k0 + kb * BK;
        if (!A_MN) {
          load_a(sa, kc, m0);
        } else {
          load_a(sa, m0, kc);
          load_a(sa + 8192, m0 + 64, kc);
        }
        if (!B_MN) {
          if (PAIR) {
            load_b(sb, kc, EPI == EPI_SWIGLU ? rank * p.F + n0 : n0 + rank * (BN / 2));
          } else if (EPI == EPI_SWIGLU) {
            load_b(sb, kc, n0);
            load_b(sb + (BN / 2) * 128, kc, p.F + n0);
          } else {
            load_b(sb, kc, n0);
          }
        } else {
          constexpr int PANELS = BN / 64;                       // of the tile
          constexpr int MINE = PAIR ? PANELS / 2 : PANELS;      // of this CTA
#pragma unroll
          for (int i = 0; i < MINE; ++i) {
            const int q = PAIR ? rank * MINE + i : i;
            int nc;
            if (EPI == EPI_SWIGLU) {
              nc = (q < PANELS / 2) ? (n0 + q * 64) : (p.F + n0 + (q - PANELS / 2) * 64);
            } else {
              nc = n0 + q * 64;
            }
            load_b(sb + i * 8192, nc, kc);
          }
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      return true;
    };
    if (!p.ep.push_on) {
      if (elect_one()) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        Tile x = fetch(walker), next;
        for (int t = walker; t < total_tiles; t += walkers, x = next) {
          next = fetch(t + walkers);
          if (!unused(x) && !load_tile(x)) break;
        }
        // The leading CTA's products release the stages of both CTAs.  The last releases, which no load waits for, have to be here
        // before this CTA may end: each stage is waited for once more (at once for one that was never used).
        if (PAIR) {
          for (int i = 0; i < STAGES && mbar_wait(&empty[stage], phase ^ 1, KID_GEMM, 5); ++i)
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    } else {
      // Push prologue active: the rows of A arrive from the peers while this kernel runs.  The whole warp walks the
      // tile list; the first time the CTA meets an expert, lane s waits (bounded) for "source s has delivered its
      // rows of this expert", then lane 0 issues the tile's loads.
      if (lane == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
      }
      const int* my_flags = reinterpret_cast<const int*>(p.ep.peers.base[p.ep.rank] + p.ep.off_flags);
      bool ok = true;
      for (int t = walker; t < total_tiles && ok; t += walkers) {
        const Tile x = fetch(t);
        const int bgroup = x.a;
        if (bgroup < 0) continue;
        if (!((s_landed[bgroup >> 5] >> (bgroup & 31)) & 1u)) {
          bool mine = true;
          if (lane < p.ep.W)
            mine = wait_flag(my_flags + bgroup * p.ep.W + lane, p.ep.epoch, p.ep.budget_ns, 9, lane, p.ep.status);
          ok = __all_sync(0xffffffffu, mine);
          if (!ok) break;
          if (lane == 0) s_landed[bgroup >> 5] |= 1u << (bgroup & 31);
          __syncwarp();
        }
        if (lane == 0) {
          fence_proxy_async_all();
          ok = load_tile(x);
        }
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the whole warp, see umma_ss_w)
    if (rank == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(PAIR ? 2 * BM : BM, BN, A_MN, B_MN);
      const uint32_t leader = elect_one() ? 1u : 0u;
      const SmemDesc dA = make_smem_desc2(smem_u32(smem), A_MN ? 8192 : 16, 1024);
      const SmemDesc dB = make_smem_desc2(smem_u32(smem) + L::A_BYTES, B_MN ? 8192 : 16, 1024);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      Tile x = fetch(walker), next;
      for (int t = walker; t < total_tiles && ok; t += walkers, x = next) {
        int k0, nkb;
        next = fetch(t + walkers);
        if (unused(x)) continue;
        krange(x, k0, nkb);
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1, KID_GEMM, 2)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(&full[stage], phase, KID_GEMM, 3, consumer_budget)) {
            if (p.ep.status && leader) atomicCAS(p.ep.status, 0, 0x10000 | (11 << 8));
            ok = false;
            break;
          }
          tc_fence_after();
          const SmemDesc a = desc_at(dA, stage * L::STAGE_BYTES), b = desc_at(dB, stage * L::STAGE_BYTES);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            const SmemDesc ak = desc_at(a, kk * (A_MN ? 2048 : 32)), bk = desc_at(b, kk * (B_MN ? 2048 : 32));
            if (PAIR) umma_ss_pair_w(leader, d_tmem, ak, bk, idesc, (kb | kk) != 0);
            else umma_ss_w(leader, d_tmem, ak, bk, idesc, (kb | kk) != 0);
          }
          if (PAIR) umma_commit_pair_w(leader, &empty[stage]);
          else umma_commit_w(leader, &empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (PAIR) umma_commit_pair_w(leader, &tfull[acc]);
        else umma_commit_w(leader, &tfull[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else if (warp < 2 + EPI_WARPS) {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    const int lane_group = warp & 3;  // TMEM lanes [32*lane_group, +32) are the ones this warp may touch
    const int col_half = (warp - 2) >> 2;  // which half of the tile's column chunks this warp stores
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    Tile x = fetch(walker), next;
    for (int t = walker; t < total_tiles && ok; t += walkers, x = next) {
      int k0, nkb;
      next = fetch(t + walkers);
      if (unused(x)) continue;
      krange(x, k0, nkb);
      const int g = x.g, nt = x.nt;
      const int row_base = x.mt * BM + lane_group * 32;
      const int row = row_base + lane;
      const bool row_ok = row < p.M;
      const uint32_t t_row = tmem_base + acc * BN + (static_cast<uint32_t>(lane_group * 32) << 16);
      const long long gbase = static_cast<long long>(g) * p.c_group_stride;
      if (!mbar_wait(&tfull[acc], acc_phase, KID_GEMM, 4, consumer_budget)) { ok = false; break; }
      tc_fence_after();
      auto release = [&]() {      // the accumulator has been read
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster(leader_addr(&tempty[acc]));
          else mbar_arrive(&tempty[acc]);
        }
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      };

      if (EPI == EPI_STORE && p.tma_out) {
        // Plain bf16 rows, 64 columns at a time: parked as bf16 (128 bytes a row, the copy engine's swizzle) and handed to the copy
        // engine, which clips at the edges of C.  An SM's ordinary stores leave at 32 bytes a clock however they are shaped, and a warp
        // that issues them waits: 2500 clocks of a tile's epilogue, which was 5000 with the decoding of the tile, against 2600 of
        // products for a grouped weight gradient at 256 rows an expert.  Before -> now: 128 of those, 2048 x 1536 and 768 x 2048,
        // 305 -> 282 and 157 -> 148 us (805 MB of results: 268 us at the 3.0 TB/s that a plain fill writes); 3000 x 4304 x 1152
        // 31 -> 27; 2048^3 18.6 -> 17; 300 x 2048 x 512 10.4 -> 8.5.
        constexpr int CH = BN / 32 / (EPI_WARPS / 4);
        const float alpha = p.alpha ? __ldg(p.alpha) : 1.f;
        uint8_t* stage_at = epi_stage + (warp - 2) * L::EPI_STAGE_BYTES;
        const uint32_t st = smem_u32(stage_at);
        const int first = nt * BN + col_half * CH * 32;
        bool held = true;
#pragma unroll 1
        for (int c = 0; c < CH; c += 2) {
          const int col0 = first + c * 32;
          if (col0 >= p.N || row_base >= p.M) break;      // uniform across the warp
          uint32_t v[2][32];
          if (nkb > 0) {
            tmem_ld_32x32b_x32(t_row + (col_half * CH + c) * 32, v[0]);
            tmem_ld_32x32b_x32(t_row + (col_half * CH + c) * 32 + 32, v[1]);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 64; ++i) v[i >> 5][i & 31] = 0u;
          }
          if (c + 2 >= CH) {
            release();
            held = false;
          }
          if (p.alpha) {
#pragma unroll
            for (int i = 0; i < 64; ++i) v[i >> 5][i & 31] = __float_as_uint(__uint_as_float(v[i >> 5][i & 31]) * alpha);
          }
          if (lane == 0) bulk_wait_read_all();      // the copy engine has read what was parked before
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int y = (8 * i + 2 * e) & 31;
              w[e] = pack_bf16(__uint_as_float(v[i >> 2][y]), __uint_as_float(v[i >> 2][y + 1]));
            }
            st_shared_v4(epi_piece_addr(st, lane, i), w[0], w[1], w[2], w[3]);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tmC, stage_at, col0, row_base, g);
            bulk_commit_group();
          }
        }
        if (held) release();
        continue;
      }
      if (EPI == EPI_STORE) {
        const int n0 = nt * BN;
        uint8_t* cbase = reinterpret_cast<uint8_t*>(p.C);
        const long long coff = gbase + static_cast<long long>(row) * p.ldc;
        constexpr int CH = BN / 32 / (EPI_WARPS / 4);
        const float alpha = p.alpha ? __ldg(p.alpha) : 1.f;
        const uint32_t st = smem_u32(epi_stage + (warp - 2) * L::EPI_STAGE_BYTES);
        // bf16 output: first element of the four rows that this lane stores in the row-major pass (null = skip it); with the scatter
        // epilogue a row goes to the rank it came from, at the entry its tag names
        auto row_dst = [&](int rr) -> __nv_bfloat16* {
          if (rr >= p.M || p.c_fp32) return nullptr;
          if (!p.ep.scat_on) return reinterpret_cast<__nv_bfloat16*>(cbase) + gbase + static_cast<long long>(rr) * p.ldc;
          const int tag = __ldcg(p.ep.row_tag + rr);
          if (tag < 0) return nullptr;
          // a tag that names no rank or no entry (rows that never landed) must not become an address
          if ((tag >> EP_TAG_SHIFT) < p.ep.W && (tag & EP_TAG_MASK) < p.ep.ret_rows)
            return reinterpret_cast<__nv_bfloat16*>(p.ep.peers.base[tag >> EP_TAG_SHIFT] + p.ep.off_ret) +
                   static_cast<long long>(tag & EP_TAG_MASK) * p.ldc;
          atomicCAS(p.ep.status, 0, 3);
          return nullptr;
        };
        if (p.ep.scat_on && p.ep.row_val && nt == 0 && col_half == 0 && row_ok) {
          const int tag = __ldcg(p.ep.row_tag + row);
          if (tag >= 0 && (tag >> EP_TAG_SHIFT) < p.ep.W && (tag & EP_TAG_MASK) < p.ep.ret_rows)
            reinterpret_cast<float*>(p.ep.peers.base[tag >> EP_TAG_SHIFT] + p.ep.off_ret_vals)[tag & EP_TAG_MASK] =
                p.ep.row_val[row];
        }
        __nv_bfloat16* rowptr[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) rowptr[j] = row_dst(row_base + (lane >> 2) + 8 * j);
#pragma unroll 1
        for (int c = col_half * CH; c < (col_half + 1) * CH; ++c) {
          const int col0 = n0 + c * 32;
          if (col0 >= p.N) break;  // uniform across the warp
          uint32_t v[32];
          if (nkb > 0) {
            tmem_ld_32x32b_x32(t_row + c * 32, v);
            tmem_ld_wait();
            if (p.alpha) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          const bool full_chunk = (col0 + 32 <= p.N);
          if (full_chunk) {
            // warp-uniform branch: every lane takes part in the transposition, rows past M are skipped on the way out; what
            // is added and the parked rows are read ahead of the first store (sums into an fp32 gradient of 128 experts, 2048 x
            // 1536 of 256 rows each: 1965 -> 822 us; every store waited for its own two loads before)
            __syncwarp();  // the previous chunk's readers are done with the staging area
            if (p.ep.scat_on) {
              // nothing is added in fp32: parked as bf16, half the shared-memory traffic (second product of 4096 tokens, one rank to itself,
              // parked as fp32 and as bf16: 128 experts, eight a token, 768 to 2048, 153 and 143 us; 16, four a token, 512 to 1024, 54 and 46)
              const int q = lane & 3;
              uint4 o[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                uint32_t w[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) w[e] = pack_bf16(__uint_as_float(v[8 * i + 2 * e]), __uint_as_float(v[8 * i + 2 * e + 1]));
                st_shared_v4(epi_piece_addr64(st, lane, i), w[0], w[1], w[2], w[3]);
              }
              __syncwarp();
#pragma unroll
              for (int j = 0; j < 4; ++j) ld_shared_v4(epi_piece_addr64(st, (lane >> 2) + 8 * j, q), o[j].x, o[j].y, o[j].z, o[j].w);
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (rowptr[j] != nullptr) *reinterpret_cast<uint4*>(rowptr[j] + col0 + 8 * q) = o[j];
              continue;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
              st_shared_v4(epi_piece_addr(st, lane, i), v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            __syncwarp();
            if (p.c_fp32) {
              const int q = lane & 7, r0 = row_base + (lane >> 3);
              float* dst = reinterpret_cast<float*>(cbase) + gbase + static_cast<long long>(r0) * p.ldc + col0 + 4 * q;
              float4 o[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                uint32_t w0, w1, w2, w3;
                ld_shared_v4(epi_piece_addr(st, (lane >> 3) + 4 * j, q), w0, w1, w2, w3);
                o[j] = make_float4(__uint_as_float(w0), __uint_as_float(w1), __uint_as_float(w2), __uint_as_float(w3));
              }
              if (p.accumulate) {
                float4 old[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  if (r0 + 4 * j < p.M) old[j] = *reinterpret_cast<const float4*>(dst + 4 * j * p.ldc);
#pragma unroll
                for (int j = 0; j < 8; ++j) { o[j].x += old[j].x; o[j].y += old[j].y; o[j].z += old[j].z; o[j].w += old[j].w; }
              }
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (r0 + 4 * j < p.M) *reinterpret_cast<float4*>(dst + 4 * j * p.ldc) = o[j];
            } else {
              const int q = lane & 3, r0 = row_base + (lane >> 2);
              __nv_bfloat16* dst[4];
              uint4 res[4], old[4];
              float f[4][8];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                dst[j] = rowptr[j];
                if (dst[j] == nullptr) continue;
                dst[j] += col0 + 8 * q;
                if (p.residual) res[j] = *reinterpret_cast<const uint4*>(p.residual + static_cast<long long>(r0 + 8 * j) * p.ldr + col0 + 8 * q);
                if (p.accumulate) old[j] = *reinterpret_cast<const uint4*>(dst[j]);
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint32_t w[8];
                ld_shared_v4(epi_piece_addr(st, (lane >> 2) + 8 * j, 2 * q), w[0], w[1], w[2], w[3]);
                ld_shared_v4(epi_piece_addr(st, (lane >> 2) + 8 * j, 2 * q + 1), w[4], w[5], w[6], w[7]);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[j][e] = __uint_as_float(w[e]);
              }
              auto add = [](float (&x)[8], const uint4& u) {
                const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c2 = unpack_bf16(u.z), d = unpack_bf16(u.w);
                x[0] += a.x; x[1] += a.y; x[2] += b.x; x[3] += b.y; x[4] += c2.x; x[5] += c2.y; x[6] += d.x; x[7] += d.y;
              };
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (dst[j] == nullptr) continue;
                if (p.residual) add(f[j], res[j]);
                if (p.accumulate) add(f[j], old[j]);
                *reinterpret_cast<uint4*>(dst[j]) = make_uint4(pack_bf16(f[j][0], f[j][1]), pack_bf16(f[j][2], f[j][3]),
                                                               pack_bf16(f[j][4], f[j][5]), pack_bf16(f[j][6], f[j][7]));
              }
            }
            continue;
          }
          if (!row_ok) continue;
          if (p.c_fp32) {
            float* dst = reinterpret_cast<float*>(cbase) + coff + col0;
#pragma unroll
            for (int i = 0; i < 32; ++i) {  // constant indices keep v[] in registers
              if (col0 + i < p.N) {
                float o = __uint_as_float(v[i]);
                if (p.accumulate) o += dst[i];
                dst[i] = o;
              }
            }
          } else {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(cbase) + coff + col0;
            const __nv_bfloat16* res = p.residual ? p.residual + static_cast<long long>(row) * p.ldr + col0 : nullptr;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (col0 + i < p.N) {
                float o = __uint_as_float(v[i]);
                if (res) o += __bfloat162float(res[i]);
                if (p.accumulate) o += __bfloat162float(dst[i]);
                dst[i] = __float2bfloat16(o);
              }
            }
          }
        }
      } else {
        // SwiGLU: accumulator columns [0,BN/2) = gate, [BN/2,BN) = up, for output columns n0..n0+BN/2.
        constexpr int HALF = BN / 2;
        const int n0 = nt * HALF;
        const float scale = (p.row_scale && row_ok) ? __ldcg(p.row_scale + row) : 1.0f;
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<long long>(row) * p.ldc;
        __nv_bfloat16* pre = p.preact ? p.preact + static_cast<long long>(row) * p.ld_preact : nullptr;
        constexpr int CH = HALF / 32 / (EPI_WARPS / 4);
#pragma unroll 1
        for (int c = col_half * CH; c < (col_half + 1) * CH; ++c) {
          const int col0 = n0 + c * 32;
          if (col0 >= p.N) break;
          uint32_t gv[32], uv[32];
          tmem_ld_32x32b_x32(t_row + c * 32, gv);
          tmem_ld_32x32b_x32(t_row + HALF + c * 32, uv);
          tmem_ld_wait();
          const int lim = min(32, p.N - col0);
          if (lim == 32) {
            // all lanes take part (warp-uniform branch): results are packed to bf16, transposed through the staging
            // area in two rounds (out + gate, then up) and stored as 64-byte row segments, 8 rows per instruction
            uint32_t o[16], pg[16], pu[16];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              // pre-activations are rounded to bf16 first so forward and backward see the same values
              float g0 = __bfloat162float(__float2bfloat16(__uint_as_float(gv[j])));
              float g1 = __bfloat162float(__float2bfloat16(__uint_as_float(gv[j + 1])));
              float u0 = __bfloat162float(__float2bfloat16(__uint_as_float(uv[j])));
              float u1 = __bfloat162float(__float2bfloat16(__uint_as_float(uv[j + 1])));
              float a0 = g0 / (1.0f + __expf(-g0)) * u0 * scale;
              float a1 = g1 / (1.0f + __expf(-g1)) * u1 * scale;
              o[j / 2] = pack_bf16(a0, a1);
              pg[j / 2] = pack_bf16(g0, g1);
              pu[j / 2] = pack_bf16(u0, u1);
            }
            const uint32_t st = smem_u32(epi_stage + (warp - 2) * L::EPI_STAGE_BYTES);
            const int q = lane & 3, r0 = row_base + (lane >> 2);
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<long long>(r0) * p.ldc + col0 + 8 * q;
            __nv_bfloat16* pdst = pre ? p.preact + static_cast<long long>(r0) * p.ld_preact + col0 + 8 * q : nullptr;
            // parked rows are read ahead of the first store of a round
            uint4 x[4], y[4];
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              st_shared_v4(epi_piece_addr64(st, lane, i), o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
              if (pre) st_shared_v4(epi_piece_addr64(st + 2048, lane, i), pg[4 * i], pg[4 * i + 1], pg[4 * i + 2], pg[4 * i + 3]);
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              ld_shared_v4(epi_piece_addr64(st, (lane >> 2) + 8 * j, q), x[j].x, x[j].y, x[j].z, x[j].w);
              if (pre) ld_shared_v4(epi_piece_addr64(st + 2048, (lane >> 2) + 8 * j, q), y[j].x, y[j].y, y[j].z, y[j].w);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (r0 + 8 * j >= p.M) continue;
              *reinterpret_cast<uint4*>(dst + 8 * j * p.ldc) = x[j];
              if (pre) *reinterpret_cast<uint4*>(pdst + 8 * j * p.ld_preact) = y[j];
            }
            if (pre) {
              __syncwarp();
#pragma unroll
              for (int i = 0; i < 4; ++i)
                st_shared_v4(epi_piece_addr64(st, lane, i), pu[4 * i], pu[4 * i + 1], pu[4 * i + 2], pu[4 * i + 3]);
              __syncwarp();
#pragma unroll
              for (int j = 0; j < 4; ++j) ld_shared_v4(epi_piece_addr64(st, (lane >> 2) + 8 * j, q), x[j].x, x[j].y, x[j].z, x[j].w);
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (r0 + 8 * j < p.M) *reinterpret_cast<uint4*>(pdst + 8 * j * p.ld_preact + p.F) = x[j];
            }
            continue;
          }
          if (!row_ok) continue;
          {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (i < lim) {
                float g0 = __bfloat162float(__float2bfloat16(__uint_as_float(gv[i])));
                float u0 = __bfloat162float(__float2bfloat16(__uint_as_float(uv[i])));
                out[col0 + i] = __float2bfloat16(g0 / (1.0f + __expf(-g0)) * u0 * scale);
                if (pre) {
                  pre[col0 + i] = __float2bfloat16(g0);
                  pre[p.F + col0 + i] = __float2bfloat16(u0);
                }
              }
            }
          }
        }
      }
      release();
    }
    if (EPI == EPI_STORE && p.tma_out && lane == 0) bulk_wait_all();
    if (p.ep.scat_on) __threadfence_system();   // this thread's peer stores are ordered before the "returned" flag
  } else if (p.ep.push_on) {
    // ------------------------------------------------------------ push warps (warps 10..11)
    // Entries are walked in send order (local expert major, owners rotated so that every owner receives from one
    // source at a time).  A warp copies PUSH_CHUNK rows, fences at system scope, then counts the rows per expert:
    // the warp whose count completes an expert raises this rank's flag for that expert on the owner.
    const EpFuse& ep = p.ep;
    const int E = ep.El * ep.W;
    const int vec = ep.H / 8;
    const bool healthy = *reinterpret_cast<volatile int*>(ep.status) == 0;
    auto flag_of = [&](int e) -> int* {
      const int o = e / ep.El;
      return reinterpret_cast<int*>(ep.peers.base[o] + ep.off_flags) + (e - o * ep.El) * ep.W + ep.rank;
    };
    if (healthy) {
      // Chunks are claimed from a counter (sent[E]) instead of being dealt out by CTA index: the owners' tiles wait for
      // rows, so every row must go out even when some CTAs of this grid are not resident yet (another kernel holds
      // their SM).  With a static split the rows of a waiting CTA would never leave while the resident CTAs spin.
      int* next_chunk = ep.sent + E;
      for (;;) {
        long long chunk = 0;
        if (lane == 0) chunk = atomicAdd(next_chunk, 1);
        chunk = __shfl_sync(0xffffffffu, chunk, 0);
        if (chunk == 0) {
          // experts this rank sends nothing to: their owners must not wait for it
          for (int e = lane; e < E; e += 32)
            if (ep.counts[e] == 0) st_release_sys(flag_of(e), ep.epoch);
        }
        const long long c0 = chunk * PUSH_CHUNK;
        if (c0 >= ep.n_entries) break;
        const int cnt = static_cast<int>(ep.n_entries - c0 < PUSH_CHUNK ? ep.n_entries - c0 : PUSH_CHUNK);
        int n_l = -1, e_l = -1, r_l = -1;
        if (lane < cnt) {
          n_l = ep.order[c0 + lane];
          if (n_l >= 0 && n_l < ep.n_entries) {   // a broken order table must not become a wild read
            e_l = ep.expert[n_l];
            r_l = ep.dest_row[n_l];
          }
        }
        for (int j = 0; j < cnt; ++j) {
          const int n = __shfl_sync(0xffffffffu, n_l, j);
          const int e = __shfl_sync(0xffffffffu, e_l, j);
          const int r = __shfl_sync(0xffffffffu, r_l, j);
          const int o = (e >= 0 && e < E) ? e / ep.El : -1;
          if (o < 0 || r < 0 || r >= ep.cap_rows) {   // never write outside the owner's buffer
            if (lane == 0) atomicExch(ep.status, 3);
            continue;
          }
          const uint4* srow = reinterpret_cast<const uint4*>(ep.src + static_cast<long long>(n / ep.k) * ep.lds);
          uint4* drow = reinterpret_cast<uint4*>(ep.peers.base[o] + ep.off_rows) + static_cast<long long>(r) * vec;
          for (int c = lane; c < vec; c += 32 * 8) {
            uint4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (c + 32 * u < vec) v[u] = srow[c + 32 * u];
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (c + 32 * u < vec) drow[c + 32 * u] = v[u];
          }
          if (lane == 0) {
            if (ep.val) reinterpret_cast<float*>(ep.peers.base[o] + ep.off_vals)[r] = ep.val[n];
            reinterpret_cast<int*>(ep.peers.base[o] + ep.off_tags)[r] = (ep.rank << EP_TAG_SHIFT) | n;
          }
        }
        __threadfence_system();
        __syncwarp();
        if (lane < cnt && e_l >= 0 && e_l < E) {
          const int before = atomicAdd(ep.sent + e_l, 1);
          if (before + 1 == ep.counts[e_l]) {
            __threadfence_system();
            st_release_sys(flag_of(e_l), ep.epoch);
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  // The other CTA's products no longer read this shared memory (both tiles' epilogues waited for them), and neither its commits
  // (drained by the producer) nor its epilogue (which arrives before it gets here) has anything left to signal on these barriers.
  if (PAIR) cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 2 * BN);
    else tmem_dealloc(tmem_base, 2 * BN);
  }
  if (p.ep.scat_on) {
    // the last CTA to get here tells every peer that this rank has returned all of its rows
    if (threadIdx.x == 0) {
      __threadfence_system();
      s_last_cta = (atomicAdd(p.ep.done_counter, 1u) == gridDim.x - 1) ? 1 : 0;
    }
    __syncthreads();
    if (s_last_cta) {
      if (static_cast<int>(threadIdx.x) < p.ep.W) {
        __threadfence_system();
        st_release_sys(reinterpret_cast<int*>(p.ep.peers.base[threadIdx.x] + p.ep.off_ret_flags) + p.ep.rank, p.ep.ret_epoch);
      }
      if (threadIdx.x == 0) *p.ep.done_counter = 0;
    }
  }
}

// ----------------------------------------------------------------------------
// Host launcher
// ----------------------------------------------------------------------------
// Host description of the expert-parallel fusion of one launch (C ABI; see `EpFuse` for the meaning of the fields).
struct EpFuseArgs {
  const unsigned long long* peer_ptrs;   // [W] base address of every rank's symmetric buffer
  int W, rank, El;
  int* status;
  long long budget_ms;
  // push prologue
  int push_on;
  long long off_rows, off_vals, off_tags, off_flags;
  const void* src;
  long long lds;
  const int* order;
  const int* expert;
  const int* dest_row;
  const float* val;
  const int* counts;
  int* sent;
  int n_entries, k, H, epoch;
  long long cap_rows;
  // scatter epilogue
  int scat_on;
  long long off_ret, off_ret_vals, off_ret_flags;
  const int* row_tag;
  const float* row_val;
  int ret_epoch;
  unsigned int* done_counter;
  int ret_rows;
};

// C (+)= alpha * sum_s ws[s] (+ residual): the second half of a split product, in a fixed order.  Four columns per thread.
__global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ ws, int splits, int M, int N, void* C, long long ldc, int c_fp32, int accumulate,
                 const __nv_bfloat16* __restrict__ residual, long long ldr, const float* __restrict__ alpha) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int nv = N / 4;
  if (idx >= static_cast<long long>(M) * nv) return;
  const long long r = idx / nv;
  const int c = static_cast<int>(idx - r * nv) * 4;
  const long long plane = static_cast<long long>(M) * N;
  const float* src = ws + r * N + c;
  float4 v = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
  for (int s = 1; s < splits; ++s) {
    const float4 u = *reinterpret_cast<const float4*>(src + s * plane);
    v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
  }
  if (alpha) { const float a = __ldg(alpha); v.x *= a; v.y *= a; v.z *= a; v.w *= a; }
  if (c_fp32) {
    float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(C) + r * ldc + c);
    if (accumulate) { const float4 o = *dst; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
    *dst = v;
  } else {
    uint2* dst = reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(C) + r * ldc + c);
    if (residual) {
      const uint2 u = *reinterpret_cast<const uint2*>(residual + r * ldr + c);
      const float2 x = unpack_bf16(u.x), y = unpack_bf16(u.y);
      v.x += x.x; v.y += x.y; v.z += y.x; v.w += y.y;
    }
    if (accumulate) {
      const uint2 u = *dst;
      const float2 x = unpack_bf16(u.x), y = unpack_bf16(u.y);
      v.x += x.x; v.y += x.y; v.z += y.x; v.w += y.y;
    }
    *dst = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
  }
}

template <int BN, bool A_MN, bool B_MN, int EPI, bool PAIR>
static int launch(const GemmArgs& a, cudaStream_t stream) {
  using L = SmemLayout<BN, PAIR>;
  CUtensorMap tmA, tmB, tmC;
  // ---- A map (2D)
  {
    uint64_t dims[2];
    uint64_t str[1] = {static_cast<uint64_t>(a.lda) * 2};
    uint32_t box[2];
    if (!A_MN) {
      // memory [M rows][K contiguous]
      dims[0] = static_cast<uint64_t>(a.K);
      dims[1] = static_cast<uint64_t>(a.M);
      box[0] = BK;
      box[1] = BM;
    } else {
      // memory [K rows][M contiguous]
      dims[0] = static_cast<uint64_t>(a.M);
      dims[1] = static_cast<uint64_t>(a.groups_k > 0 ? a.total_rows : a.K);
      box[0] = 64;
      box[1] = BK;
    }
    int r = make_tmap_bf16(&tmA, a.A, 2, dims, str, box);
    if (r) return 10000 + r;
  }
  // ---- B map (3D, last dim = group)
  const int n_mem = (EPI == EPI_SWIGLU) ? 2 * a.F : a.N;
  {
    uint64_t dims[3];
    uint64_t str[2];
    uint32_t box[3];
    str[0] = static_cast<uint64_t>(a.ldb) * 2;
    const uint64_t rows_b = !B_MN ? static_cast<uint64_t>(n_mem)
                                  : static_cast<uint64_t>(a.groups_k > 0 ? a.total_rows : a.K);
    str[1] = a.b_groups > 1 ? static_cast<uint64_t>(a.b_group_stride) * 2 : rows_b * str[0];
    dims[2] = static_cast<uint64_t>(a.b_groups > 1 ? a.b_groups : 1);
    if (!B_MN) {
      // memory [N rows][K contiguous]
      dims[0] = static_cast<uint64_t>(a.K);
      dims[1] = rows_b;
      box[0] = BK;
      box[1] = (EPI == EPI_SWIGLU || PAIR) ? BN / 2 : BN;
    } else {
      // memory [K rows][N contiguous]
      dims[0] = static_cast<uint64_t>(n_mem);
      dims[1] = rows_b;
      box[0] = 64;
      box[1] = BK;
    }
    box[2] = 1;
    int r = make_tmap_bf16(&tmB, a.B, 3, dims, str, box);
    if (r) return 20000 + r;
  }
  GemmParams p;
  memset(&p.ep, 0, sizeof(p.ep));
  if (a.ep) {
    const EpFuseArgs& e = *a.ep;
    for (int i = 0; i < MAX_RANKS; ++i) p.ep.peers.base[i] = i < e.W ? e.peer_ptrs[i] : 0ull;
    p.ep.W = e.W; p.ep.rank = e.rank; p.ep.El = e.El; p.ep.status = e.status;
    p.ep.budget_ns = static_cast<unsigned long long>(e.budget_ms) * 1000000ull;
    p.ep.push_on = e.push_on;
    p.ep.off_rows = e.off_rows; p.ep.off_vals = e.off_vals; p.ep.off_tags = e.off_tags; p.ep.off_flags = e.off_flags;
    p.ep.src = reinterpret_cast<const __nv_bfloat16*>(e.src); p.ep.lds = e.lds;
    p.ep.order = e.order; p.ep.expert = e.expert; p.ep.dest_row = e.dest_row; p.ep.val = e.val;
    p.ep.counts = e.counts; p.ep.sent = e.sent;
    p.ep.n_entries = e.n_entries; p.ep.k = e.k; p.ep.H = e.H; p.ep.epoch = e.epoch; p.ep.cap_rows = e.cap_rows;
    p.ep.scat_on = e.scat_on;
    p.ep.off_ret = e.off_ret; p.ep.off_ret_vals = e.off_ret_vals; p.ep.off_ret_flags = e.off_ret_flags;
    p.ep.row_tag = e.row_tag; p.ep.row_val = e.row_val; p.ep.ret_epoch = e.ret_epoch;
    p.ep.done_counter = e.done_counter;
    p.ep.ret_rows = e.ret_rows;
  }
  p.M = a.M; p.N = a.N; p.K = a.K;
  constexpr int TN = (EPI == EPI_SWIGLU) ? BN / 2 : BN;
  constexpr int TM = PAIR ? 2 * BM : BM;
  p.m_tiles = a.tile_group ? a.m_tiles_cap : (a.M + TM - 1) / TM;
  p.n_tiles = (a.N + TN - 1) / TN;
  p.groups_k = a.groups_k;
  p.C = a.C; p.ldc = a.ldc; p.c_group_stride = a.c_group_stride;
  p.c_fp32 = a.c_fp32; p.accumulate = a.accumulate;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(a.residual); p.ldr = a.ldr;
  p.tile_group = a.tile_group; p.group_rows = a.group_rows;
  p.F = a.F; p.row_scale = a.row_scale; p.alpha = a.alpha;
  p.preact = reinterpret_cast<__nv_bfloat16*>(a.preact); p.ld_preact = a.ld_preact;
  p.k_splits = 1; p.kb_per_split = 0;
  const bool split = a.split_ws != nullptr && a.k_splits > 1;
  if (split) {
    const int nkb = (a.K + BK - 1) / BK;
    p.kb_per_split = (nkb + a.k_splits - 1) / a.k_splits;
    p.k_splits = (nkb + p.kb_per_split - 1) / p.kb_per_split;     // every piece has at least one k-block
    p.C = a.split_ws; p.ldc = a.N; p.c_group_stride = static_cast<long long>(a.M) * a.N;
    p.c_fp32 = 1; p.accumulate = 0; p.residual = nullptr; p.alpha = nullptr;
  }

  const long long total = static_cast<long long>(p.m_tiles) * p.n_tiles * (p.groups_k > 0 ? p.groups_k : p.k_splits);
  if (total <= 0) return 0;
  if (total >= (1ll << 31) - 65536) return 910;
  // ---- C map (3D, last dim = group)
  tmC = tmA;       // placeholder where nothing is stored through it
  p.tma_out = EPI == EPI_STORE && !split && !a.c_fp32 && !a.residual && !a.accumulate && !p.ep.scat_on && a.M > 0 && a.N > 0 &&
              (a.groups_k == 0 || a.c_group_stride % 8 == 0);
  if (p.tma_out) {
    const uint64_t dims[3] = {static_cast<uint64_t>(a.N), static_cast<uint64_t>(a.M), static_cast<uint64_t>(a.groups_k > 0 ? a.groups_k : 1)};
    const uint64_t str[2] = {static_cast<uint64_t>(a.ldc) * 2, static_cast<uint64_t>(a.groups_k > 0 ? a.c_group_stride : a.ldc * a.M) * 2};
    const uint32_t box[3] = {64, 32, 1};
    int r = make_tmap_bf16(&tmC, a.C, 3, dims, str, box);
    if (r) return 30000 + r;
  }
  constexpr int RASTER_M = PAIR ? 8 : 16;
  p.by_group = fast_div(p.m_tiles * p.n_tiles);
  p.by_band = fast_div(RASTER_M * p.n_tiles);
  p.by_rest = fast_div(p.m_tiles % RASTER_M ? p.m_tiles % RASTER_M : 1);

  auto kfn = gemm_kernel<BN, A_MN, B_MN, EPI, PAIR>;
  static bool smem_done[16] = {};
  {
    const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kfn), L::TOTAL, smem_done);
    if (e != cudaSuccess) return 300 + static_cast<int>(e);
  }
  if (PAIR) {
    const int pairs = static_cast<int>(total < a.num_sms / 2 ? total : a.num_sms / 2);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = L::TOTAL;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kfn, tmA, tmB, tmC, p);
    if (e != cudaSuccess) return 400 + static_cast<int>(e);
  } else {
    const int grid = static_cast<int>(total < a.num_sms ? total : a.num_sms);
    kfn<<<grid, p.ep.push_on ? GEMM_THREADS_PUSH : GEMM_THREADS, L::TOTAL, stream>>>(tmA, tmB, tmC, p);
  }
  if (split) {
    const long long n = static_cast<long long>(a.M) * (a.N / 4);
    split_sum_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(
        a.split_ws, p.k_splits, a.M, a.N, a.C, a.ldc, a.c_fp32, a.accumulate, reinterpret_cast<const __nv_bfloat16*>(a.residual), a.ldr,
        a.alpha);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + static_cast<int>(e);
}

// Whether two CTAs share a 256-row tile (wide products whose tiles are all of one problem).  Each then loads half of B for twice
// the rows: a third less traffic into shared memory and out of L2, and less power for it, which under the power cap is clock.
// Measured, one CTA per 128-row tile -> pairs: 8192^3 748 -> 712 us; 8192 x 24576 x 4096 with SwiGLU 1130 -> 1072;
// 4096 x 151936 x 2048 1762 -> 1594; 24576 x 4096 x 8192 (both operands across rows) 1097 -> 1036; 4096 x 5120 x 2048 68 -> 64.
// Where the line lies:
//  * a tile of 256 rows can waste half of itself at M's end: the waves decide, one of pairs costing at most 0.95 of a single one
//    (300 x 32000 x 512, four waves of pairs against three: 21 -> 27 us);
//  * short runs do not make up for the handshakes between the two at the first loads and the last stores: 32 k-blocks per CTA
//    (2048^3) 21 -> 23 us, 47 (3456 x 1152 x 3000) the same, 68 (3000 x 1152 x 4304) 39 -> 35;
//  * grouped weight gradients have few k-blocks per tile (four at 256 rows per expert), so a tile is mostly its epilogue, and the
//    epilogue of one half waits for the other's: 128 x 2048 x 1536 and 128 x 768 x 2048 of 256 rows 282 -> 300 and 148 -> 176;
//  * experts' rows in 256-row tiles: an odd number of 128-row tiles leaves half a pair idle, which takes back what the shared loads
//    save (128 experts of 256 rows on average 250 -> 257, of exactly 192 rows 213 -> 198).
static bool pays_in_pairs(const GemmArgs& a) {
  if (a.tile_group || a.ep || a.groups_k > 0 || a.M <= BM || a.num_sms < 2) return false;
  const long long nt = a.epi == EPI_SWIGLU ? (a.N + 127) / 128 : (a.N + 255) / 256;
  const int splits = a.split_ws && a.k_splits > 1 ? a.k_splits : 1, pairs = a.num_sms / 2;
  const long long one = ((a.M + BM - 1) / BM * nt * splits + a.num_sms - 1) / a.num_sms;                // waves
  const long long two = ((a.M + 2 * BM - 1) / (2 * BM) * nt * splits + pairs - 1) / pairs;
  const long long kb = (static_cast<long long>(a.K) + BK - 1) / BK / splits;
  return 19 * two <= 20 * one && one * kb >= 48;
}

}  // namespace ttb

// Returns 0 on success; non-zero codes: 10000+r / 20000+r tensor-map encode failure of A / B (r = CUresult),
// 300+e shared-memory opt-in, 400+e launch (e = cudaError_t), 9xx bad arguments.
TTB_EXPORT int ttb_gemm_bf16(const ttb::GemmArgs* args, void* stream_ptr) {
  using namespace ttb;
  const GemmArgs& a = *args;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  if ((a.lda % 8) || (a.ldb % 8)) return 901;
  if ((reinterpret_cast<uintptr_t>(a.A) | reinterpret_cast<uintptr_t>(a.B)) & 15) return 902;
  // vectorised epilogue stores: 16-byte aligned rows
  if (a.c_fp32 ? (a.ldc % 4) : (a.ldc % 8)) return 903;
  if (reinterpret_cast<uintptr_t>(a.C) & 15) return 903;
  if (a.residual && ((a.ldr % 8) || (reinterpret_cast<uintptr_t>(a.residual) & 15))) return 904;
  if (a.epi == EPI_SWIGLU && ((a.F % 8) || a.c_fp32 || (a.preact && (a.ld_preact % 8)))) return 905;
  if (a.alpha && a.epi != EPI_STORE) return 905;
  if (a.split_ws && (a.epi != EPI_STORE || a.tile_group || a.groups_k > 0 || a.ep || (a.N % 8) || (reinterpret_cast<uintptr_t>(a.split_ws) & 15)))
    return 909;
  if (a.ep) {
    const EpFuseArgs& e = *a.ep;
    if (!a.tile_group || a.groups_k > 0 || e.W < 1 || e.W > MAX_RANKS || e.El < 1 || e.El * e.W > 1024 || !e.status) return 906;
    if (e.push_on && (a.a_mn || (e.H % 8) || (e.lds % 8) || !e.order || !e.expert || !e.dest_row || !e.counts || !e.sent ||
                      e.n_entries < 0 || e.n_entries > EP_TAG_MASK || (e.off_rows % 16)))
      return 907;
    // the scatter epilogue lives in the bf16 row-major store path: whole 32-column chunks, no residual / accumulate
    if (e.scat_on && (a.epi != EPI_STORE || a.c_fp32 || a.accumulate || a.residual || (a.N % 32) || !e.row_tag ||
                      !e.done_counter || (e.off_ret % 16)))
      return 908;
  }
  const bool wide = (a.epi == EPI_SWIGLU) ? true : (a.N > 128);
  const bool pair = wide && pays_in_pairs(a);
#define TTB_DISPATCH(AMN, BMN)                                                                                            \
  if (a.epi == EPI_SWIGLU)                                                                                                \
    return pair ? launch<256, AMN, BMN, EPI_SWIGLU, true>(a, stream) : launch<256, AMN, BMN, EPI_SWIGLU, false>(a, stream); \
  if (wide) return pair ? launch<256, AMN, BMN, EPI_STORE, true>(a, stream) : launch<256, AMN, BMN, EPI_STORE, false>(a, stream); \
  return launch<128, AMN, BMN, EPI_STORE, false>(a, stream);
  if (!a.a_mn && !a.b_mn) { TTB_DISPATCH(false, false) }
  if (!a.a_mn && a.b_mn) { TTB_DISPATCH(false, true) }
  if (a.a_mn && a.b_mn) { TTB_DISPATCH(true, true) }
  if (a.a_mn && !a.b_mn) { TTB_DISPATCH(true, false) }
#undef TTB_DISPATCH
  return 999;
}

TTB_EXPORT int ttb_gemm_status(unsigned int* out4, int reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out4, ttb::g_status_word, sizeof(unsigned int) * 4);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (reset) {
    unsigned int z[4] = {0, 0, 0, 0};
    e = cudaMemcpyToSymbol(ttb::g_status_word, z, sizeof(z));
  }
  return static_cast<int>(e);
}
