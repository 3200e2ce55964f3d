// Entry points that the launch sequences (layers.cu) and the C++ nodes (nodes.cpp) call.  The sources that define them include
// this file too, so that a signature that drifts apart does not compile.  What they do stands at the definitions.
#pragma once
#include <cuda_runtime_api.h>

extern "C" {
// elementwise.cu, gemm.cu, attention.cu, moe.cu
int b2_rmsnorm_fwd(const void* x, const void* delta, const float* w, void* sum_out, void* y, float* rstd, int rows, int D,
                   float eps, int* status, cudaStream_t s);
int b2_rmsnorm_bwd(const void* dy, const void* x, const float* w, const float* rstd, const void* residual, void* dx,
                   float* dw_partial, float* dw, int rows, int D, int* status, cudaStream_t s);
int b2_gemm_nt(const void* a, const void* w, void* d, int M, int N, int K, long long lda, long long ldw, long long ldd,
               int num_experts, const int* tile_expert, const int* num_m_tiles, int group_align256, int epi, int* status,
               cudaStream_t stream);
int b2_gemm_nt_rope(const void* a, const void* w, void* d, int M, int N, int K, long long lda, long long ldd, const float* cos_t,
                    const float* sin_t, int rope_cols, int seq, int* status, cudaStream_t stream);
int b2_gemm_nn(const void* a, const void* w, const void* w2, void* d, int M, int N, int K, int k_split, long long lda,
               long long ldw, long long ldd, int num_experts, const int* tile_expert, const int* num_m_tiles, int group_align256,
               const float* alpha, int* status, cudaStream_t stream);
int b2_gemm_tn(const void* a, const void* b, void* d, void* d2, int m_split, int M, int N, int R, long long lda, long long ldb,
               long long ldd, int num_experts, const int* expert_offsets, const int* expert_counts, int out_kind, float beta,
               const float* alpha, int* status, cudaStream_t stream);
int b2_gemm_swiglu(const void* a, const void* w1, const void* w3, void* h, void* gate, void* up, int M, int F, int K,
                   long long lda, int num_experts, const int* tile_expert, const int* num_m_tiles, int group_align256,
                   int* status, cudaStream_t stream);
int b2_gemm_nn_swiglu_bwd(const void* a, const void* w, const void* gate, const void* up, void* dgu, void* h, int M, int F, int K,
                          long long lda, int num_experts, const int* tile_expert, const int* num_m_tiles, int group_align256,
                          int* status, cudaStream_t stream);
int b2_swiglu_bwd(const void* dh, const void* gate, const void* up, void* dgu, void* h, const int* live_rows, int rows, int F,
                  cudaStream_t s);
int b2_attention_fwd_ex(const void* q, const void* k, const void* v, long long q_pitch, long long k_pitch, long long v_pitch,
                        void* out, float* lse, int B, int S, int Hq, int Hkv, float scale, int causal, int f16, int* status,
                        cudaStream_t stream);
int b2_attention_bwd_rope(const void* dout, const void* q, const void* k, const void* v, const void* out, const float* lse,
                          long long q_pitch, long long k_pitch, long long v_pitch, float* stats, void* dq, void* dk, void* dv,
                          long long dq_pitch, long long dk_pitch, long long dv_pitch, int B, int S, int Hq, int Hkv, float scale,
                          int causal, const float* rope_cos, const float* rope_sin, int* status, cudaStream_t stream);
int b2_cross_entropy2(void* logits, const long long* targets, void* loss, int wide, int T, int V, float loss_scale,
                      float grad_scale, int* status, cudaStream_t s);
int b2_router_fwd(const void* x, const void* w, float* weights, long long* idx, float* probs, int T, int N, int K, cudaStream_t s);
int b2_skinny_tn(const float* dy, const void* x, float* dw, int T, int N, int K, cudaStream_t s);
int b2_moe_plan(const long long* idx, int slots, int E, int* slot_row, int* row_slot, int* offs, int* tile_expert, int* meta,
                int* counts, int capacity_rows, cudaStream_t s);
int b2_moe_gather(const void* x, const int* row_slot, const int* meta, const float* scale, const void* y_perm, float* dweights,
                  void* x_perm, int D, int capacity_rows, int slots, cudaStream_t s);
int b2_moe_combine(const void* y_perm, const int* slot_row, const float* weights, const void* residual, void* out, int T, int D,
                   int rows, cudaStream_t s);
int b2_moe_dx(const void* dy, const int* slot_row, const float* dweights, const float* probs, const long long* idx,
              const float* weights, const float* daux, const int* counts, const void* w, float* dlogits, void* dx, int T, int N,
              int D, int rows, cudaStream_t s);
int b2_rmsnorm_bwd_parts(int rows, int D);
int b2_scale_bf16(void* x, const float* factor, long long n, cudaStream_t s);
int b2_embedding_fwd(const long long* ids, const void* table, void* out, int T, int D, cudaStream_t s);
int b2_embedding_bwd(const long long* ids, const void* dy, float* dtable, int T, int D, cudaStream_t s);
int b2_moe_aux(const float* probs, const int* counts, float* aux, int T, int E, cudaStream_t s);
// layers.cu
const char* b2_layers_refused();
int b2_attn_half_fwd(const void* x, const float* ln1, const void* wqkv, const float* cos_t, const float* sin_t, const void* wo,
                     const float* ln2, void* n1, void* qkv, void* a, void* proj, void* sum, void* n2, float* stats, int B, int S,
                     int Hq, int Hkv, float eps1, float eps2, int* status, cudaStream_t s);
int b2_attn_half_bwd(const void* dsum, const void* dn2, const void* x, const float* ln1, const void* wqkv, const float* cos_t,
                     const float* sin_t, const void* wo, const float* ln2, const void* n1, const void* qkv, const void* a,
                     const void* sum, const float* stats, float* gqkv, float* go, float* dln1, float* dln2, void* dx, void* dmid,
                     void* da, void* dn1, void* dqkv, float* partial, float* row_stats, int B, int S, int Hq, int Hkv, int* status,
                     cudaStream_t s);
int b2_moe_layer_fwd(const void* x, const void* router, const void* w1, const void* w3, const void* w2, const void* residual,
                     float* weights, long long* idx, float* probs, int* tables, void* x_perm, void* h, void* gate, void* up,
                     void* y_perm, void* out, int T, int D, int F, int E, int cap, int* status, cudaStream_t s);
int b2_swiglu_bwd_in_product(long long M, int F, int K);
int b2_head_chunk(const void* hidden, const void* weight, const long long* targets, void* logits, double* loss, void* dh,
                  float* grad, int T, int V, int D, float loss_scale, float grad_scale, int* status, cudaStream_t s);
int b2_moe_experts_bwd(const void* dout, const void* w1, const void* w3, const void* w2, const float* weights, int* tables,
                       const void* x_perm, const void* y_perm, void* gate, void* up, int rebuild, void* g1, void* g3, void* g2,
                       int expert_kind, void* dy_perm, void* dgu, void* h, void* dh, void* dx_perm, float* dweights, int T, int D,
                       int F, int E, int cap, int* status, cudaStream_t s);
int b2_moe_router_bwd(const void* x, const void* router, const float* weights, const long long* idx, const float* probs,
                      int* tables, const float* daux, float* grouter, const void* dx_perm, const float* dweights, float* dlogits,
                      void* dx, int T, int D, int E, int cap, cudaStream_t s);
}
