// C entry points that csrc/host.cpp calls and the argument structure of the GEMM, declared once for both sides: every kernel source
// includes this (through common.cuh), so a definition whose parameters differ from what the launch functions pass does not compile.
#pragma once
#include <cuda_bf16.h>

#define TTB_EXPORT extern "C" __attribute__((visibility("default")))

namespace ttb {

struct EpFuseArgs;   // gemm.cu

struct GemmArgs {
  const void* A;      // bf16
  long long lda;      // elements: row stride of A's memory matrix
  const void* B;      // bf16
  long long ldb;      // elements: row stride of B's memory matrix
  long long b_group_stride;  // elements between B[g] (grouped-M), 0 otherwise
  int b_groups;       // number of B groups (>=1)
  void* C;
  long long ldc;
  long long c_group_stride;
  int M, N, K;        // grouped-K: K ignored, M = rows of A^T ( = columns of A memory ), N = cols of B memory
  int a_mn, b_mn;     // memory orientation: 0 = K contiguous, 1 = M/N contiguous
  int c_fp32, accumulate;
  const void* residual;
  long long ldr;
  const int* tile_group;
  int m_tiles_cap;    // grouped-M: number of m tiles to schedule (capacity)
  const int* group_rows;
  int groups_k;
  long long total_rows;  // grouped-K: total rows of A/B memory matrices
  int epi;            // 0 store, 1 swiglu
  int F;
  const float* row_scale;
  void* preact;
  long long ld_preact;
  int num_sms;
  const EpFuseArgs* ep;          // optional expert-parallel fusion (grouped-M launches only)
  const float* alpha;            // optional device scalar multiplied into the product (plain stores only)
  float* split_ws;               // optional fp32 [k_splits, M, N]: the product is formed in k_splits pieces, then added up
  int k_splits;
};

// inputs of the chunk-parallel delta-rule kernels (delta_chunk.cuh)
struct DeltaChunkIn {
  const __nv_bfloat16 *q, *k, *v;                      // row r, head h, channel c at [r * *_t + h * *_h + c]
  long long q_t, q_h, k_t, k_h, v_t, v_h;
  const float *g, *beta;                               // log decay [rows, H] or [rows, H, 128]; step size [rows, H]
  const int* chunk_rows;                               // [NC, 3]: first row, rows (1 .. 64), sequence
  int H, NC, l2;
  float scale;
  int rep;                                             // value heads per key head: head h reads q and k of head h / rep
};

}  // namespace ttb

TTB_EXPORT int ttb_gemm_bf16(const ttb::GemmArgs*, void*);
TTB_EXPORT int ttb_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, float*, long long, int, float, int, void*);
TTB_EXPORT int ttb_rmsnorm_bwd(const void*, const void*, const void*, const float*, const void*, void*, float*, void*, int, long
                            long, int, int, int, void*);
TTB_EXPORT int ttb_layernorm_fwd(const void*, const void*, const void*, void*, float*, float*, long long, int, float, void*);
TTB_EXPORT int ttb_layernorm_bwd(const void*, const void*, const void*, const float*, const float*, void*, float*, void*, int,
                            long long, int, int, void*);
TTB_EXPORT int ttb_bias_act_fwd(const void*, const void*, const void*, void*, long long, int, int, void*);
TTB_EXPORT int ttb_bias_act_bwd(const void*, const void*, const void*, void*, float*, void*, int, long long, int, int, int,
                            void*);
TTB_EXPORT int ttb_qknorm_rope_fwd(const void*, long long, int, int, int, const void*, const void*, const float*, const float*,
                            void*, void*, float*, long long, float, int, void*);
TTB_EXPORT int ttb_qknorm_rope_bwd(const void*, const void*, const void*, const void*, long long, int, int, int, const void*,
                            const void*, const float*, const float*, const float*, void*, long long, float*, void*, int, long
                            long, int, int, void*);
TTB_EXPORT int ttb_delta_prep(const ttb::DeltaChunkIn*, float*, float*, float*, void*, void*, float*, void*);
TTB_EXPORT int ttb_delta_out(const ttb::DeltaChunkIn*, const float*, const float*, const float*, int, void*, void*);
TTB_EXPORT int ttb_delta_bwd_pre(const ttb::DeltaChunkIn*, const void*, const float*, int, float*, float*, void*);
TTB_EXPORT int ttb_delta_vec_prep(const ttb::DeltaChunkIn*, float*, float*, float*, void*, void*, float*, void*);
TTB_EXPORT int ttb_delta_vec_out(const ttb::DeltaChunkIn*, const float*, const float*, const float*, int, void*, void*);
TTB_EXPORT int ttb_delta_vec_bwd_pre(const ttb::DeltaChunkIn*, const void*, const float*, int, float*, float*, void*);
TTB_EXPORT int ttb_delta_state_scan(const void*, const void*, const float*, float*, const float*, int, const float*, const float*, float*,
                            const int*, int, int, int, int, int, float, float, void*);
TTB_EXPORT int ttb_scale(const void*, int, const float*, void*, int, long long, int, void*);
TTB_EXPORT int ttb_copy_words(void*, const void*, long long, void*);
TTB_EXPORT int ttb_kda_gate_row_blocks(long long, int);
TTB_EXPORT int ttb_kda_gate_fwd(const void*, const void*, int, const void*, int, float*, long long, int, int, float, void*);
TTB_EXPORT int ttb_kda_gate_bwd(const float*, const void*, const void*, int, const void*, int, void*, float*, float*, long long, int, int, float,
                            void*);
TTB_EXPORT int ttb_gdn_gate_fwd(const void*, long long, const void*, long long, const void*, int, const void*, int, float*, float*, long long,
                            int, void*);
TTB_EXPORT int ttb_gdn_gate_bwd(const float*, const float*, const void*, long long, const void*, int, const void*, int, const float*, void*,
                            void*, float*, void*, int, long long, int, int, void*);
TTB_EXPORT int ttb_qkv_rope_fwd(const void*, const void*, const float*, const float*, void*, void*, void*, long long, int, int, int, void*);
TTB_EXPORT int ttb_qkv_rope_bwd(const void*, const void*, const void*, const float*, const float*, void*, float*, void*, int, long long, int,
                            int, int, void*);
TTB_EXPORT int ttb_rope(const void*, long long, long long, const float*, const float*, void*, long long, int, int, float,
                            void*);
TTB_EXPORT int ttb_swiglu_fwd(const void*, long long, void*, long long, const float*, long long, int, const int*, void*);
TTB_EXPORT int ttb_swiglu_bwd(const void*, long long, const void*, long long, const float*, void*, long long, float*, void*,
                            long long, long long, int, const int*, void*);
TTB_EXPORT int ttb_attn_fwd(const void*, long long, const void*, long long, const void*, long long, void*, float*, float*, const
                            int*, int, int, long long, int, int, int, int, float, int, void*);
TTB_EXPORT int ttb_attn_bwd(const void*, const void*, long long, const void*, long long, const void*, const void*, const float*,
                            float*, float*, float*, float*, void*, void*, void*, const int*, int, long long, int, int, int, int,
                            float, int, int, void*);
TTB_EXPORT int ttb_attn_bwd_dq(const void*, const void*, long long, const void*, long long, const void*, const float*, const
                            float*, void*, const int*, int, long long, int, int, int, int, float, int, void*);
