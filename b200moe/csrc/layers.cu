// Whole layers as one call: the launches of a block's attention half and of a routed layer, forward and backward, in the order
// in which the separate operations issue them, with the same kernels and the same choices.  What a small layer costs is the
// host: an operation takes some 25 us from Python (arguments, allocations, autograd) beside 2-3 us for the launch itself, so a
// training step of two blocks of width 512 spent 4.7 ms on 1.5 ms of kernels.
//
// Every entry point returns 0, or the code of the first launch that was refused (b2_layers_refused: its entry point).  Buffers
// are the caller's.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "entries.h"

typedef __nv_bfloat16 bf16;

namespace {
// The launch that was refused last in this thread.
thread_local const char* refused = "";

// Calls one after the other; stops at the first that is refused.
struct Sequence {
  int rc = 0;
  template <typename F> void operator()(const char* name, F call) {
    if (rc == 0 && (rc = call()) != 0) refused = name;
  }
};
// The routing tables of one layer, laid out one behind the other (moe_plan's outputs).
struct Tables {
  int *slot_row, *row_slot, *offs, *tile_expert, *meta, *counts;
  Tables(int* base, int slots, int cap, int E)
      : slot_row(base), row_slot(slot_row + slots), offs(row_slot + cap), tile_expert(offs + E), meta(tile_expert + cap / 128),
        counts(meta + 4) {}
};
constexpr float HEAD_SCALE = 0.08838834764831845f;      // 128^-1/2
}  // namespace

extern "C" {

const char* b2_layers_refused() { return refused; }

// Attention half of a block: n1 = rmsnorm(x); qkv = n1 Wqkv^T with q and k rotated; a = causal attention; sum = x + a Wo^T;
// n2 = rmsnorm(sum).  T = B S rows of D = 128 Hq columns; qkv has 128 (Hq + 2 Hkv).  stats: fp32, T reciprocal deviations of
// x, T of sum, then the attention's B Hq S log-sum-exps.  proj: scratch [T, D].
int b2_attn_half_fwd(const void* x, const float* ln1, const void* wqkv, const float* cos_t, const float* sin_t, const void* wo,
                     const float* ln2, void* n1, void* qkv, void* a, void* proj, void* sum, void* n2, float* stats, int B, int S,
                     int Hq, int Hkv, float eps1, float eps2, int* status, cudaStream_t s) {
  const int T = B * S, D = Hq * 128, N = (Hq + 2 * Hkv) * 128;
  bf16* const q = static_cast<bf16*>(qkv);
  Sequence run;
  run("b2_rmsnorm_fwd", [&] { return b2_rmsnorm_fwd(x, nullptr, ln1, nullptr, n1, stats, T, D, eps1, status, s); });
  run("b2_gemm_nt_rope", [&] {
    return b2_gemm_nt_rope(n1, wqkv, qkv, T, N, D, D, N, cos_t, sin_t, (Hq + Hkv) * 128, S, status, s);
  });
  run("b2_attention_fwd_ex", [&] {
    return b2_attention_fwd_ex(q, q + Hq * 128, q + (Hq + Hkv) * 128, N, N, N, a, stats + 2 * static_cast<size_t>(T), B, S, Hq, Hkv,
                               HEAD_SCALE, 1, 0, status, s);
  });
  run("b2_gemm_nt", [&] { return b2_gemm_nt(a, wo, proj, T, D, D, D, D, D, 1, nullptr, nullptr, 0, 0, status, s); });
  run("b2_rmsnorm_fwd", [&] { return b2_rmsnorm_fwd(x, proj, ln2, sum, n2, stats + T, T, D, eps2, status, s); });
  return run.rc;
}

// Its backward pass: dx for the gradients dsum and dn2; the weights' gradients are added to gqkv and go (fp32), the gains' are
// stored to dln1 and dln2 (fp32 [D]).  Scratch: dmid, da, dn1 [T, D], dqkv [T, N], partial fp32 (rmsnorm_bwd's),
// row_stats fp32 [B Hq, 2, S].  dn1 may be da, and dmid may be dx (see b2_rmsnorm_bwd).
int b2_attn_half_bwd(const void* dsum, const void* dn2, const void* x, const float* ln1, const void* wqkv, const float* cos_t,
                     const float* sin_t, const void* wo, const float* ln2, const void* n1, const void* qkv, const void* a,
                     const void* sum, const float* stats, float* gqkv, float* go, float* dln1, float* dln2, void* dx, void* dmid,
                     void* da, void* dn1, void* dqkv, float* partial, float* row_stats, int B, int S, int Hq, int Hkv, int* status,
                     cudaStream_t s) {
  const int T = B * S, D = Hq * 128, N = (Hq + 2 * Hkv) * 128;
  const bf16* const q = static_cast<const bf16*>(qkv);
  bf16* const dq = static_cast<bf16*>(dqkv);
  Sequence run;
  run("b2_rmsnorm_bwd", [&] { return b2_rmsnorm_bwd(dn2, sum, ln2, stats + T, dsum, dmid, partial, dln2, T, D, status, s); });
  run("b2_gemm_nn", [&] {
    return b2_gemm_nn(dmid, wo, nullptr, da, T, D, D, 0, D, D, D, 1, nullptr, nullptr, 0, nullptr, status, s);
  });
  run("b2_gemm_tn", [&] {
    return b2_gemm_tn(dmid, a, go, nullptr, 0, D, D, T, D, D, D, 1, nullptr, nullptr, 1, 1.f, nullptr, status, s);
  });
  run("b2_attention_bwd_rope", [&] {
    return b2_attention_bwd_rope(da, q, q + Hq * 128, q + (Hq + Hkv) * 128, a, stats + 2 * static_cast<size_t>(T), N, N, N, row_stats,
                                 dq, dq + Hq * 128, dq + (Hq + Hkv) * 128, N, N, N, B, S, Hq, Hkv, HEAD_SCALE, 1, cos_t, sin_t,
                                 status, s);
  });
  run("b2_gemm_nn", [&] {
    return b2_gemm_nn(dqkv, wqkv, nullptr, dn1, T, D, N, 0, N, D, D, 1, nullptr, nullptr, 0, nullptr, status, s);
  });
  run("b2_gemm_tn", [&] {
    return b2_gemm_tn(dqkv, n1, gqkv, nullptr, 0, N, D, T, N, D, D, 1, nullptr, nullptr, 1, 1.f, nullptr, status, s);
  });
  run("b2_rmsnorm_bwd", [&] { return b2_rmsnorm_bwd(dn1, x, ln1, stats, dmid, dx, partial, dln1, T, D, status, s); });
  return run.rc;
}

// Routed layer on one rank: router, plan, gather, gate/up product with SwiGLU, down projection, combine (+ residual).  gate and
// up are null where nothing is kept for a backward pass; h is scratch.
int b2_moe_layer_fwd(const void* x, const void* router, const void* w1, const void* w3, const void* w2, const void* residual,
                     float* weights, long long* idx, float* probs, int* tables, void* x_perm, void* h, void* gate, void* up,
                     void* y_perm, void* out, int T, int D, int F, int E, int cap, int* status, cudaStream_t s) {
  const Tables t(tables, 2 * T, cap, E);
  Sequence run;
  run("b2_router_fwd", [&] { return b2_router_fwd(x, router, weights, idx, probs, T, E, D, s); });
  run("b2_moe_plan", [&] {
    return b2_moe_plan(idx, 2 * T, E, t.slot_row, t.row_slot, t.offs, t.tile_expert, t.meta, t.counts, cap, s);
  });
  run("b2_moe_gather", [&] { return b2_moe_gather(x, t.row_slot, t.meta, nullptr, nullptr, nullptr, x_perm, D, cap, 2 * T, s); });
  run("b2_gemm_swiglu", [&] {
    return b2_gemm_swiglu(x_perm, w1, w3, h, gate, up, cap, F, D, D, E, t.tile_expert, t.meta, 1, status, s);
  });
  run("b2_gemm_nt", [&] { return b2_gemm_nt(h, w2, y_perm, cap, D, F, F, F, D, E, t.tile_expert, t.meta, 1, 0, status, s); });
  run("b2_moe_combine", [&] { return b2_moe_combine(y_perm, t.slot_row, weights, residual, out, T, D, cap, s); });
  return run.rc;
}

// Whether the SwiGLU backward of M rows of F columns behind a reduction over K rides in the product (see
// b200moe.ops.native.gemm_nn_swiglu_bwd, which has the figures).
int b2_swiglu_bwd_in_product(long long M, int F, int K) { return K >= 2048 || M * F <= 1 << 21; }

// One chunk of tokens through the LM head: logits = hidden W^T become their own gradient (and the loss is added to the double
// ``loss``), dh = dlogits W, grad (fp32) += dlogits^T hidden.
int b2_head_chunk(const void* hidden, const void* weight, const long long* targets, void* logits, double* loss, void* dh,
                  float* grad, int T, int V, int D, float loss_scale, float grad_scale, int* status, cudaStream_t s) {
  Sequence run;
  run("b2_gemm_nt", [&] { return b2_gemm_nt(hidden, weight, logits, T, V, D, D, D, V, 1, nullptr, nullptr, 0, 0, status, s); });
  run("b2_cross_entropy2", [&] { return b2_cross_entropy2(logits, targets, loss, 1, T, V, loss_scale, grad_scale, status, s); });
  run("b2_gemm_nn", [&] {
    return b2_gemm_nn(logits, weight, nullptr, dh, T, D, V, 0, V, D, D, 1, nullptr, nullptr, 0, nullptr, status, s);
  });
  run("b2_gemm_tn", [&] {
    return b2_gemm_tn(logits, hidden, grad, nullptr, 0, V, D, T, V, D, D, 1, nullptr, nullptr, 1, 1.f, nullptr, status, s);
  });
  return run.rc;
}

// Backward pass of the routed layer, the experts: dx_perm and dweights [T, 2] for the output's gradient; those of w1, w3, w2 are
// added to g1, g3, g2 (expert_kind 1: fp32, 2: bf16).  rebuild: gate and up are scratch and are formed again.  dh: scratch
// [cap, F] where the SwiGLU backward is a kernel of its own, null where it rides in the product.  Scratch besides: dy_perm
// [cap, D], dgu [cap, 2F], h [cap, F].  dx_perm [cap, D] may overlap dh, and gate and up where they are scratch: it is stored
// behind the kernels that read them.
int b2_moe_experts_bwd(const void* dout, const void* w1, const void* w3, const void* w2, const float* weights, int* tables,
                       const void* x_perm, const void* y_perm, void* gate, void* up, int rebuild, void* g1, void* g3, void* g2,
                       int expert_kind, void* dy_perm, void* dgu, void* h, void* dh, void* dx_perm, float* dweights, int T, int D,
                       int F, int E, int cap, int* status, cudaStream_t s) {
  const Tables t(tables, 2 * T, cap, E);
  Sequence run;
  if (rebuild)
    run("b2_gemm_swiglu", [&] {
      return b2_gemm_swiglu(x_perm, w1, w3, h, gate, up, cap, F, D, D, E, t.tile_expert, t.meta, 1, status, s);
    });
  run("b2_moe_gather", [&] {
    return b2_moe_gather(dout, t.row_slot, t.meta, weights, y_perm, dweights, dy_perm, D, cap, 2 * T, s);
  });
  if (dh) {
    run("b2_gemm_nn", [&] {
      return b2_gemm_nn(dy_perm, w2, nullptr, dh, cap, F, D, 0, D, F, F, E, t.tile_expert, t.meta, 1, nullptr, status, s);
    });
    run("b2_swiglu_bwd", [&] { return b2_swiglu_bwd(dh, gate, up, dgu, h, t.meta + 1, cap, F, s); });
  } else {
    run("b2_gemm_nn_swiglu_bwd", [&] {
      return b2_gemm_nn_swiglu_bwd(dy_perm, w2, gate, up, dgu, h, cap, F, D, D, E, t.tile_expert, t.meta, 1, status, s);
    });
  }
  run("b2_gemm_nn", [&] {
    return b2_gemm_nn(dgu, w1, w3, dx_perm, cap, D, 2 * F, F, 2 * F, D, D, E, t.tile_expert, t.meta, 1, nullptr, status, s);
  });
  run("b2_gemm_tn", [&] {
    return b2_gemm_tn(dy_perm, h, g2, nullptr, 0, D, F, cap, D, F, F, E, t.offs, t.counts, expert_kind, 1.f, nullptr, status, s);
  });
  run("b2_gemm_tn", [&] {
    return b2_gemm_tn(dgu, x_perm, g1, g3, F, 2 * F, D, cap, 2 * F, D, D, E, t.offs, t.counts, expert_kind, 1.f, nullptr, status, s);
  });
  return run.rc;
}

// Its router, behind the experts (whose scratch the caller may have given back): dx [T, D]; the gradient of the router's weights
// is added to grouter (fp32).  Scratch: dlogits [T, E].
int b2_moe_router_bwd(const void* x, const void* router, const float* weights, const long long* idx, const float* probs,
                      int* tables, const float* daux, float* grouter, const void* dx_perm, const float* dweights, float* dlogits,
                      void* dx, int T, int D, int E, int cap, cudaStream_t s) {
  const Tables t(tables, 2 * T, cap, E);
  Sequence run;
  run("b2_moe_dx", [&] {
    return b2_moe_dx(dx_perm, t.slot_row, dweights, probs, idx, weights, daux, t.counts, router, dlogits, dx, T, E, D, cap, s);
  });
  run("b2_skinny_tn", [&] { return b2_skinny_tn(dlogits, x, grouter, T, E, D, s); });
  return run.rc;
}

}  // extern "C"
