// Expert-routing kernels for one GPU's share of the MoE block: the dispatch plan
// (a stable counting sort of the (token, j) slots by expert, computed by one CTA
// with no host round trip), the row gather into the padded expert-major layout,
// the weighted combine and their backward duals.
//
// Layout contract.  Slots are numbered s = 2*token + j.  Expert e owns rows
// [seg_start[e], seg_start[e] + count[e]) of the permuted buffer, in slot order;
// every segment is padded with zero rows to a multiple of 256 so a GEMM tile
// never straddles two experts.  ``slot_row[s]`` is the row of slot s,
// ``row_slot[r]`` the slot of row r (-1 for padding), ``offs[e]`` the padded
// cumulative segment ends, ``tile_expert[i]`` the expert of 128-row tile i and
// ``meta = {live tiles, live rows}``.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "chain.cuh"
#include "debug.cuh"
#include "entries.h"
#include "ptx.cuh"

namespace b2 {

constexpr int PLAN_THREADS = 1024;
constexpr int ALIGN_ROWS = 256;   // segment padding; tile tables are per 128-row unit
constexpr int TILE_ROWS = 128;
constexpr int PLAN_CLUSTER_SLOTS = 2560;      // from here on eight CTAs plan (2048 slots 5.0 us on one, 5.3 on eight; 3000 6.1, 5.4)

// One CTA, or a cluster of eight for many slots: a warp owns a run of slots, reads 32 of them at a time (coalesced) and ranks
// those of one expert among its lanes by ballots; counts per warp and expert are scanned between the counting and the placing
// pass, those of the CTAs through the cluster's shared memory.  Bound by latency, and from some thousand slots on by what one
// SM can issue (32768 slots 28 us on one CTA).  us before, when a thread owned a run of its own and a scan over 1024 threads
// followed for every expert, and now: 2048 slots 5.1, 5.0; 8192 18, 5.6; 32768 84, 7.9.
__global__ void __launch_bounds__(PLAN_THREADS) moe_plan_kernel(const long long* __restrict__ idx, int slots, int E,
                                                                int* __restrict__ slot_row, int* __restrict__ row_slot,
                                                                int* __restrict__ offs, int* __restrict__ tile_expert,
                                                                int* __restrict__ meta, int* __restrict__ counts_out,
                                                                int capacity_rows) {
  chain_begin();
  extern __shared__ int plan_smem[];
  constexpr int WARPS = PLAN_THREADS / 32, AHEAD = 8;
  int* const at = plan_smem;                  // [WARPS][E] counts, then the next row of each warp and expert
  int* const seg_count = at + WARPS * E;      // [E]
  int* const seg_start = seg_count + E;       // [E + 1]
  int* const cta_count = seg_start + E + 1;   // [E] slots of this CTA
  int* const cta_first = cta_count + E;       // [E] slots of the CTAs before it
  uint32_t ctas;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(ctas));
  const int rank = static_cast<int>(cluster_ctarank());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* const mine = at + warp * E;
  const int all_warps = WARPS * static_cast<int>(ctas), my_warp = rank * WARPS + warp;
  const int per = ((slots + all_warps - 1) / all_warps + 31) / 32 * 32;
  const int s0 = min(slots, my_warp * per), s1 = min(slots, s0 + per);

  for (int i = tid; i < WARPS * E; i += PLAN_THREADS) at[i] = 0;
  __syncthreads();
  // visits the warp's slots 32 at a time: (slot, expert, lanes of the same expert), E for lanes behind the last slot
  auto visit = [&](auto&& body) {
    for (int first = s0; first < s1; first += 32 * AHEAD) {
      int e[AHEAD];
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        const int s = first + i * 32 + lane;
        e[i] = s < s1 ? min(max(static_cast<int>(idx[s]), 0), E - 1) : E;
      }
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        if (first + i * 32 >= s1) break;
        unsigned same = 0xffffffffu;          // lanes whose expert has the same bits (a match instruction takes longer)
        for (int bit = 0; E >> bit; ++bit) {
          const unsigned ones = __ballot_sync(0xffffffffu, e[i] >> bit & 1);
          same &= e[i] >> bit & 1 ? ones : ~ones;
        }
        body(first + i * 32 + lane, e[i], same);
      }
    }
  };
  visit([&](int, int e, unsigned same) {
    if (e < E && lane == __ffs(same) - 1) mine[e] += __popc(same);
    __syncwarp();
  });
  __syncthreads();
  for (int e = warp; e < E; e += WARPS) {     // exclusive scan over the warps
    const int count = at[lane * E + e];
    int inc = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += up;
    }
    at[lane * E + e] = inc - count;
    if (lane == 31) {
      cta_count[e] = seg_count[e] = inc;
      cta_first[e] = 0;
    }
  }
  if (ctas > 1) cluster_sync_all();
  else __syncthreads();
  for (int e = tid; ctas > 1 && e < E; e += PLAN_THREADS) {
    int total = 0, before = 0;
    for (int r = 0; r < static_cast<int>(ctas); ++r) {
      int count;
      asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(count) : "r"(mapa_u32(smem_u32(cta_count + e), r)) : "memory");
      total += count;
      if (r < rank) before += count;
    }
    seg_count[e] = total;
    cta_first[e] = before;
  }
  if (ctas > 1) __syncthreads();
  if (tid == 0) {
    int row = 0;
    for (int e = 0; e < E; ++e) {
      seg_start[e] = row;
      row += (seg_count[e] + ALIGN_ROWS - 1) / ALIGN_ROWS * ALIGN_ROWS;
      if (rank == 0) {
        offs[e] = row;
        if (counts_out) counts_out[e] = seg_count[e];
      }
    }
    seg_start[E] = row;
    if (rank == 0) {
      meta[0] = row / TILE_ROWS;
      meta[1] = row;
      meta[2] = row > capacity_rows ? 1 : 0;   // overflow flag (cannot happen with capacity = slots + E*255)
    }
  }
  __syncthreads();
  for (int e = my_warp; e < E; e += all_warps) {     // tiles and padding rows of an expert
    const int begin = seg_start[e], end = seg_start[e + 1];
    for (int t = begin / TILE_ROWS + lane; t < min(end, capacity_rows) / TILE_ROWS; t += 32) tile_expert[t] = e;
    for (int r = begin + seg_count[e] + lane; r < min(end, capacity_rows); r += 32) row_slot[r] = -1;
  }
  visit([&](int s, int e, unsigned same) {
    if (e < E) {
      const int row = seg_start[e] + cta_first[e] + mine[e] + __popc(same & ((1u << lane) - 1));
      slot_row[s] = row;
      if (row < capacity_rows) row_slot[row] = s;
    }
    __syncwarp();
    if (e < E && lane == __ffs(same) - 1) mine[e] += __popc(same);
    __syncwarp();
  });
  if (ctas > 1) cluster_sync_all();           // the others have read this CTA's counts
}

struct alignas(16) vec16 {
  uint32_t v[4];
};

// x_perm[r] = scale(slot) * x[slot / 2] for live rows, zeros for padding; one warp per row.
// ``scale`` is null (dispatch) or the per-slot routing weight (backward of combine).
// With ``y_perm``/``dweights`` the kernel also emits dweights[slot] = <x[token], y_perm[r]>.
__global__ void __launch_bounds__(256) moe_gather_kernel(const __nv_bfloat16* __restrict__ x,
                                                         const int* __restrict__ row_slot,
                                                         const int* __restrict__ meta,
                                                         const float* __restrict__ scale,
                                                         const __nv_bfloat16* __restrict__ y_perm,
                                                         float* __restrict__ dweights,
                                                         __nv_bfloat16* __restrict__ x_perm, int D, int capacity_rows,
                                                         int slots) {
  chain_begin();
  const int live_rows = min(meta[1], capacity_rows);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = blockIdx.x * 8 + warp; r < live_rows; r += gridDim.x * 8) {
    const int slot = row_slot[r];
    __nv_bfloat16* dst = x_perm + static_cast<size_t>(r) * D;
    if (slot < 0) {
      for (int c = lane * 8; c < D; c += 256) *reinterpret_cast<vec16*>(dst + c) = vec16{{0, 0, 0, 0}};
      continue;
    }
    if (!dbg_in_range(slot, 0, slots, 411)) continue;
    const __nv_bfloat16* src = x + static_cast<size_t>(slot >> 1) * D;
    if (!scale) {
      for (int c = lane * 8; c < D; c += 256) *reinterpret_cast<vec16*>(dst + c) = *reinterpret_cast<const vec16*>(src + c);
      continue;
    }
    const float w = scale[slot];
    float dot = 0.f;
    for (int c = lane * 8; c < D; c += 256) {
      const vec16 in = *reinterpret_cast<const vec16*>(src + c);
      vec16 yv{{0, 0, 0, 0}};
      if (y_perm) yv = *reinterpret_cast<const vec16*>(y_perm + static_cast<size_t>(r) * D + c);
      vec16 out;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&in.v[i]));
        const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&yv.v[i]));
        dot += f.x * g.x + f.y * g.y;
        const __nv_bfloat162 o = __floats2bfloat162_rn(f.x * w, f.y * w);
        out.v[i] = *reinterpret_cast<const uint32_t*>(&o);
      }
      *reinterpret_cast<vec16*>(dst + c) = out;
    }
    if (dweights) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (lane == 0) dweights[slot] = dot;
    }
  }
}

// out[t] = (residual[t] +) w0 * y[slot_row[2t]] + w1 * y[slot_row[2t+1]]   (weights null => 1); one warp per token.
// The weighted sum is rounded to bf16 before the residual is added: the layer's output followed by the block's sum, bit
// for bit (a router further on turns another rounding into another choice between experts that are nearly tied).
__global__ void __launch_bounds__(256) moe_combine_kernel(const __nv_bfloat16* __restrict__ y_perm,
                                                          const int* __restrict__ slot_row,
                                                          const float* __restrict__ weights,
                                                          const __nv_bfloat16* __restrict__ residual,
                                                          __nv_bfloat16* __restrict__ out, int T, int D, int rows) {
  chain_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = blockIdx.x * 8 + warp; t < T; t += gridDim.x * 8) {
    const int r0 = slot_row[2 * t], r1 = slot_row[2 * t + 1];
    if (!dbg_in_range(r0, 0, rows, 412) || !dbg_in_range(r1, 0, rows, 412)) continue;
    const float w0 = weights ? weights[2 * t] : 1.f, w1 = weights ? weights[2 * t + 1] : 1.f;
    const __nv_bfloat16* a = y_perm + static_cast<size_t>(r0) * D;
    const __nv_bfloat16* b = y_perm + static_cast<size_t>(r1) * D;
    for (int c = lane * 8; c < D; c += 256) {
      const vec16 va = *reinterpret_cast<const vec16*>(a + c);
      const vec16 vb = *reinterpret_cast<const vec16*>(b + c);
      vec16 vr{{0, 0, 0, 0}};
      if (residual) vr = *reinterpret_cast<const vec16*>(residual + static_cast<size_t>(t) * D + c);
      vec16 o;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&va.v[i]));
        const float2 fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&vb.v[i]));
        __nv_bfloat162 r = __floats2bfloat162_rn(__fmaf_rn(w1, fb.x, w0 * fa.x), __fmaf_rn(w1, fb.y, w0 * fa.y));
        if (residual) {
          const float2 fr = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&vr.v[i]));
          const float2 f = __bfloat1622float2(r);
          r = __floats2bfloat162_rn(fr.x + f.x, fr.y + f.y);
        }
        o.v[i] = *reinterpret_cast<const uint32_t*>(&r);
      }
      *reinterpret_cast<vec16*>(out + static_cast<size_t>(t) * D + c) = o;
    }
  }
}

// Balance loss of top-2 routing, E * sum_e (counts[e] / A) * (sum_t probs[t,e]) * (2 / A) with A = 2 T assignments, one
// CTA: a short reduction over T x E probabilities.  (As PyTorch operations: some twenty launches forward and backward
// per layer, and a bincount that waits for the device.)
__device__ __forceinline__ float aux_factor(int T, int E) {
  const float assignments = fmaxf(2.f * T, 1.f);
  return E * 2.f / (assignments * assignments);
}
__global__ void __launch_bounds__(1024) moe_aux_kernel(const float* __restrict__ probs, const int* __restrict__ counts,
                                                       float* __restrict__ aux, int T, int E) {
  chain_begin();
  __shared__ float partial[32];
  float sum = 0.f;
  const long long total = static_cast<long long>(T) * E;
  // a thread's stride is a multiple of E, so it stays in one column
  const int threads = 1024 / E * E;
  if (static_cast<int>(threadIdx.x) < threads) {
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
    long long i = threadIdx.x;
    for (; i + 3LL * threads < total; i += 4LL * threads) {
      s0 += probs[i];
      s1 += probs[i + threads];
      s2 += probs[i + 2LL * threads];
      s3 += probs[i + 3LL * threads];
    }
    for (; i < total; i += threads) s0 += probs[i];
    sum = ((s0 + s1) + (s2 + s3)) * counts[threadIdx.x % E];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x < 32) {
    sum = partial[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (threadIdx.x == 0) *aux = sum * aux_factor(T, E);
  }
}

// Input gradient of a routed layer on one GPU, in one launch:
//   dlogits[t] = backward of softmax, top-2 and renormalisation for dweights[t]
//                (+ daux * d(balance loss)/dlogits[t], which needs the probabilities and the experts' slot counts only)
//   dx[t] = dy[slot_row[2t]] + dy[slot_row[2t+1]] + dlogits[t] Wr
// Memory bound (two rows read, one written per token).  A warp works on four tokens at a time, so that an unpacked
// router weight (shared memory) serves four of them.  Router backward, its input gradient, the combine and the sum of
// the two gradients were four launches, 121 us at 5003 tokens of width 4096 inside a pass; this one takes 73.
constexpr int DX_TOKENS = 4;
template <int NN>
__global__ void __launch_bounds__(256) moe_dx_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ slot_row,
                                                     const float* __restrict__ dweights,
                                                     const float* __restrict__ probs, const long long* __restrict__ idx,
                                                     const float* __restrict__ weights,
                                                     const float* __restrict__ daux, const int* __restrict__ counts,
                                                     const __nv_bfloat16* __restrict__ w, float* __restrict__ dlogits,
                                                     __nv_bfloat16* __restrict__ dx, int T, int N, int D, int rows) {
  chain_begin();
  extern __shared__ __nv_bfloat16 dx_ws[];
  __shared__ float grads[8][DX_TOKENS][NN];
  for (int i = threadIdx.x * 8; i < N * D; i += blockDim.x * 8)
    *reinterpret_cast<vec16*>(dx_ws + i) = *reinterpret_cast<const vec16*>(w + i);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float aux_scale = daux ? *daux * aux_factor(T, N) : 0.f;
  for (int t0 = (blockIdx.x * 8 + warp) * DX_TOKENS; t0 < T; t0 += gridDim.x * 8 * DX_TOKENS) {
    if (lane < DX_TOKENS && t0 + lane < T) {
      const size_t t = t0 + lane;
      const int a = min(max(static_cast<int>(idx[2 * t]), 0), N - 1), b = min(max(static_cast<int>(idx[2 * t + 1]), 0), N - 1);
      const float da = dweights[2 * t], db = dweights[2 * t + 1];
      const float pa = probs[t * N + a], pb = probs[t * N + b];
      const float s = pa + pb;
      const float inner = da * weights[2 * t] + db * weights[2 * t + 1];
      const float dpa = (da - inner) / s, dpb = (db - inner) / s;
      const float dot = dpa * pa + dpb * pb;
      float balance = 0.f;
      if (daux)
        for (int e = 0; e < N; ++e) balance += counts[e] * probs[t * N + e];
      for (int e = 0; e < N; ++e) {
        const float dp = e == a ? dpa : (e == b ? dpb : 0.f);
        const float p = probs[t * N + e];
        float g = p * (dp - dot);
        if (daux) g += aux_scale * p * (counts[e] - balance);
        grads[warp][lane][e] = g;
        dlogits[t * N + e] = g;
      }
    }
    __syncwarp();
    const __nv_bfloat16* first[DX_TOKENS];
    const __nv_bfloat16* second[DX_TOKENS];
    float d[DX_TOKENS][NN];
#pragma unroll
    for (int j = 0; j < DX_TOKENS; ++j) {
      const int t = min(t0 + j, T - 1);
      int r0 = slot_row[2 * t], r1 = slot_row[2 * t + 1];
      if (!dbg_in_range(r0, 0, rows, 413)) r0 = 0;
      if (!dbg_in_range(r1, 0, rows, 413)) r1 = 0;
      first[j] = dy + static_cast<size_t>(r0) * D;
      second[j] = dy + static_cast<size_t>(r1) * D;
#pragma unroll
      for (int n = 0; n < NN; ++n) d[j][n] = n < N && t0 + j < T ? grads[warp][j][n] : 0.f;
    }
    for (int k = lane * 8; k < D; k += 256) {
      vec16 va[DX_TOKENS], vb[DX_TOKENS];
#pragma unroll
      for (int j = 0; j < DX_TOKENS; ++j) {
        va[j] = *reinterpret_cast<const vec16*>(first[j] + k);
        vb[j] = *reinterpret_cast<const vec16*>(second[j] + k);
      }
      float2 o[DX_TOKENS][4];
#pragma unroll
      for (int j = 0; j < DX_TOKENS; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&va[j].v[i]));
          const float2 fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&vb[j].v[i]));
          o[j][i] = make_float2(fa.x + fb.x, fa.y + fb.y);
        }
#pragma unroll
      for (int n = 0; n < NN; ++n) {
        if (n < N) {
          const vec16 wv = *reinterpret_cast<const vec16*>(dx_ws + n * D + k);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&wv.v[i]));
#pragma unroll
            for (int j = 0; j < DX_TOKENS; ++j) {
              o[j][i].x += d[j][n] * f.x;
              o[j][i].y += d[j][n] * f.y;
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < DX_TOKENS; ++j) {
        if (t0 + j >= T) continue;
        vec16 out;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 r = __floats2bfloat162_rn(o[j][i].x, o[j][i].y);
          out.v[i] = *reinterpret_cast<const uint32_t*>(&r);
        }
        *reinterpret_cast<vec16*>(dx + static_cast<size_t>(t0 + j) * D + k) = out;
      }
    }
    __syncwarp();
  }
}

}  // namespace b2

using namespace b2;
typedef __nv_bfloat16 bf16;

static int sm_count_moe() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return sms;
}

extern "C" {

// idx: int64 [slots] expert of each slot.  Outputs int32: slot_row [slots], row_slot [capacity_rows],
// offs [E], tile_expert [capacity_rows/128], meta [4], counts (optional) [E].
int b2_moe_plan(const long long* idx, int slots, int E, int* slot_row, int* row_slot, int* offs, int* tile_expert,
                int* meta, int* counts, int capacity_rows, cudaStream_t s) {
  if (E < 1) return -10;
  // 49 experts are what an earlier form of the kernel held in shared memory; this one needs 144 bytes an expert.  The limit
  // stays what callers and tests know.
  if (E > 49) return -11;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = slots >= PLAN_CLUSTER_SLOTS ? 8 : 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3(attr[1].val.clusterDim.x);
  cfg.blockDim = dim3(PLAN_THREADS);
  cfg.dynamicSmemBytes = static_cast<size_t>(E) * (PLAN_THREADS / 32) * 4 + (4 * E + 1) * 4;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = slots >= PLAN_CLUSTER_SLOTS ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, moe_plan_kernel, idx, slots, E, slot_row, row_slot, offs, tile_expert, meta, counts,
                         capacity_rows) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return 0;
}

int b2_moe_gather(const void* x, const int* row_slot, const int* meta, const float* scale, const void* y_perm,
                  float* dweights, void* x_perm, int D, int capacity_rows, int slots, cudaStream_t s) {
  if (D % 8) return -10;
  launch_next(moe_gather_kernel, sm_count_moe() * 8, 256, 0, s, (const bf16*)x, row_slot, meta, scale, (const bf16*)y_perm,
              dweights, (bf16*)x_perm, D, capacity_rows, slots);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b2_moe_combine(const void* y_perm, const int* slot_row, const float* weights, const void* residual, void* out,
                   int T, int D, int rows, cudaStream_t s) {
  if (D % 8) return -10;
  launch_next(moe_combine_kernel, min((T + 7) / 8, sm_count_moe() * 8), 256, 0, s, (const bf16*)y_perm, slot_row, weights,
              (const bf16*)residual, (bf16*)out, T, D, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// probs fp32 [T,E], counts int32 [E] -> aux, one fp32 value.
int b2_moe_aux(const float* probs, const int* counts, float* aux, int T, int E, cudaStream_t s) {
  if (E < 1 || E > 1024) return -10;
  launch_next(moe_aux_kernel, 1, 1024, 0, s, probs, counts, aux, T, E);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// See moe_dx_kernel.  N <= 16 experts; daux (device scalar: gradient of the balance loss) and counts may be null.
int b2_moe_dx(const void* dy, const int* slot_row, const float* dweights, const float* probs, const long long* idx,
              const float* weights, const float* daux, const int* counts, const void* w, float* dlogits, void* dx, int T,
              int N, int D, int rows, cudaStream_t s) {
  if (N < 2 || N > 16 || D % 8) return -10;
  const size_t smem = static_cast<size_t>(N) * D * 2;
  if (smem > 200 * 1024) return -11;
  static bool set = false;
  if (!set) {
    cudaFuncSetAttribute(moe_dx_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(moe_dx_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    set = true;
  }
  auto kernel = N <= 8 ? moe_dx_kernel<8> : moe_dx_kernel<16>;
  launch_next(kernel, min((T + 31) / 32, sm_count_moe() * 2), 256, smem, s, (const bf16*)dy, slot_row, dweights, probs, idx,
              weights, daux, counts, (const bf16*)w, dlogits, (bf16*)dx, T, N, D, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // extern "C"

B2_DEFINE_DEBUG_READER(b2_moe_debug_read)
