// Launchers that one source defines and another calls: both include this file, so that a changed parameter list does not compile in one of them.
#pragma once
#include "host_util.h"

constexpr int FF_SKINNY_MAX_ROWS = 128;        // most rows of the products of gemm_skinny.cu

// gemm_skinny.cu
FF_EXPORT int ff_gemm_skinny_plan(int M, int N, int K, long long* scratch_bytes, long long* counter_bytes);
FF_EXPORT int ff_gemm_skinny_plan_epi(int M, int N, int K, int epi, long long* scratch_bytes, long long* counter_bytes);
FF_EXPORT int ff_gemm_skinny(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw, int ldy, int grid, float* scratch, int* counters,
                             int* status, cudaStream_t stream);
FF_EXPORT int ff_gemm_skinny_swiglu(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw, int ldy, int grid, float* scratch, int* counters,
                                    int gate, float limit, int* status, cudaStream_t stream);
FF_EXPORT int ff_gemm_skinny_rope_kv(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw, int ldy, int grid, float* scratch, int* counters,
                                     const float* cos_sin, const int* slots, void* kcache, void* vcache, int hq, int hkv, int rot_dim, int block_size,
                                     int num_blocks, int* status, cudaStream_t stream);

// attention_tc.cu
FF_EXPORT int ff_attn_prefill_tc(const void* q, const void* kcache, const void* vcache, const int* block_table, const int* q_start, const int* q_lens,
                                 const int* ctx_lens, void* out, int batch, int total_rows, int max_q_len, int hq, int hkv, int dk, int dv, int ldq, int ldo,
                                 int max_blocks, int num_blocks, float scale, int window, int chunk, const float* sinks, const void* gate, int ldg, int ldv,
                                 int keep, float softcap, const void* head_gate, int ldhg, int* status, cudaStream_t s);

// norm_embed.cu
FF_EXPORT int ff_add_rmsnorm(const void* x, void* res, const void* w, void* out, void* capture, int capture_stride, int rows, int hidden, int ldx, float eps,
                             int unit_offset, int* status, cudaStream_t s);
