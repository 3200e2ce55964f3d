// Memory-bound kernels of the training step: RMSNorm (with fused residual add),
// router (skinny GEMV, softmax/top-2 and their backward), SwiGLU backward,
// cross-entropy (in-place gradient), AdamW, embedding, RoPE.
// bf16 activations move as 16-byte vectors; all arithmetic is fp32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "chain.cuh"
#include "entries.h"
#include "ptx.cuh"

namespace b2 {

struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float total = 0.f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) total += scratch[i];
  return total;
}
template <int THREADS>
__device__ __forceinline__ float block_max(float v, float* scratch) {
  v = warp_max(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float total = -INFINITY;
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) total = fmaxf(total, scratch[i]);
  return total;
}

// ------------------------------------------------------------------ RMSNorm
// Both directions are bound by memory traffic.  Eight warps work on the rows, W of them on one row (so that narrow rows keep
// every lane busy: 512 columns are one warp's), a ninth brings blocks of 8 / W consecutive rows into a ring in shared memory
// by bulk copies: the next blocks arrive while the present one is reduced, whatever the registers hold.  us, one CTA per row
// with loads through registers -> now: backward with residual and column sum 1024 x 512 11.9 -> 6.2, 4096 x 1024 22 -> 14,
// 16384 x 4096 164 -> 109 (4.9 TB/s); forward 16384 x 4096 72 -> 53, with the sum 123 -> 98.
constexpr int NORM_THREADS = 256;      // the warps that work on the rows
constexpr int NORM_VECS = 2;           // 16-byte vectors of a row per thread, 4 beyond 4096 columns
constexpr int NORM_MAX_D = 8192;
constexpr int NORM_RING = 4;

struct NormBars {
  uint64_t full[NORM_RING], empty[NORM_RING];
};

// The producer warp: blocks ``blockIdx.x``, ``+ gridDim.x``, ... of up to R rows of each tensor (null ones are left out).
template <int R, int TENSORS>
__device__ __forceinline__ void norm_producer(const __nv_bfloat16* const (&src)[TENSORS], uint8_t* ring, int ring_stages,
                                              NormBars& bars, int* status, int rows, int D) {
  if ((threadIdx.x & 31) != 0) return;
  const int blocks = (rows + R - 1) / R;
  const uint32_t row_bytes = D * 2, slot = R * row_bytes;
  int count = 0;
  for (int block = blockIdx.x; block < blocks; block += gridDim.x, ++count) {
    const int s = count % ring_stages;
    if (!mbar_wait(&bars.empty[s], ((count / ring_stages) & 1) ^ 1)) {
      atomicExch(status, 6);
      break;
    }
    const uint32_t bytes = min(R, rows - block * R) * row_bytes;
    uint32_t tensors = 0;
#pragma unroll
    for (int i = 0; i < TENSORS; ++i) tensors += src[i] != nullptr;
    mbar_expect_tx(&bars.full[s], tensors * bytes);
#pragma unroll
    for (int i = 0; i < TENSORS; ++i)
      if (src[i])
        bulk_load(ring + (static_cast<size_t>(s) * TENSORS + i) * slot, src[i] + static_cast<size_t>(block) * R * D, &bars.full[s],
                  bytes);
  }
  // copies of a CTA whose other warps gave up land before it exits
  for (int i = max(0, count - ring_stages); i < count; ++i) mbar_wait(&bars.full[i % ring_stages], (i / ring_stages) & 1);
}

__device__ __forceinline__ void norm_init(NormBars& bars) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < NORM_RING; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], NORM_THREADS / 32);
    }
    mbar_fence_init();
  }
  __syncthreads();
}

// Waits for a block.  A warp whose wait ran out reports and goes on without waiting: the warps of a row meet at barriers.
__device__ __forceinline__ bool norm_arrived(bool so_far, uint64_t& bar, uint32_t parity, int* status) {
  if (!so_far) return false;
  if (mbar_wait(&bar, parity)) return true;
  if ((threadIdx.x & 31) == 0) atomicExch(status, 6);
  return false;
}

// Sum over one row, whose W warps hold V x 256 columns each: the sums of 256 (W = 8: of the V parts of a thread together)
// columns are formed by shuffles and added in the order of the columns.  ``scratch`` alternates between two halves, so that
// one barrier per row is enough.
template <int W, int V>
__device__ __forceinline__ float norm_row_sum(float (&part)[V], float (*scratch)[8], int slot, int warp_in_row, int lane) {
  if (W == 8) {
    float v = part[0];
    v = warp_sum(v);
    if (lane == 0) scratch[0][warp_in_row] = v;
  } else {
#pragma unroll
    for (int c = 0; c < V; ++c) part[c] = warp_sum(part[c]);
    if (W == 1) {
      float total = 0.f;
#pragma unroll
      for (int c = 0; c < V; ++c) total += part[c];
      return total;
    }
    if (lane == 0) {
#pragma unroll
      for (int c = 0; c < V; ++c) scratch[slot][c * W + warp_in_row] = part[c];
    }
  }
  asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(W * 32) : "memory");
  float total = 0.f;
#pragma unroll
  for (int i = 0; i < (W == 8 ? 8 : W * V); ++i) total += scratch[slot][i];
  return total;
}

// y = (x [+ delta]) * rstd * w ; optionally writes the sum.
template <int W, int V>
__global__ void __launch_bounds__(NORM_THREADS + 32) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                                       const __nv_bfloat16* __restrict__ delta,
                                                                       const float* __restrict__ w,
                                                                       __nv_bfloat16* __restrict__ sum_out,
                                                                       __nv_bfloat16* __restrict__ y,
                                                                       float* __restrict__ rstd, int* __restrict__ status,
                                                                       int rows, int D, float eps, int ring_stages) {
  chain_begin();
  constexpr int R = 8 / W;
  extern __shared__ __align__(128) uint8_t norm_ring[];
  __shared__ NormBars bars;
  __shared__ float scratch[2][R][8];
  norm_init(bars);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == NORM_THREADS / 32) {
    const __nv_bfloat16* const src[2] = {x, delta};
    norm_producer<R, 2>(src, norm_ring, ring_stages, bars, status, rows, D);
    return;
  }
  const int slot = warp / W, in_row = warp % W;
  float wv[V][8];
#pragma unroll
  for (int c = 0; c < V; ++c) {
    const int col = ((c * W + in_row) * 32 + lane) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) wv[c][i] = col < D ? w[col + i] : 0.f;
  }
  const int blocks = (rows + R - 1) / R;
  int count = 0;
  bool here = true;
  for (int block = blockIdx.x; block < blocks; block += gridDim.x, ++count) {
    const int s = count % ring_stages;
    const int row = block * R + slot;
    const bool live = row < rows;
    const size_t base = static_cast<size_t>(row) * D;
    const __nv_bfloat16* in = reinterpret_cast<const __nv_bfloat16*>(norm_ring) + (static_cast<size_t>(s) * 2 * R + slot) * D;
    here = norm_arrived(here, bars.full[s], (count / ring_stages) & 1, status);
    bf16x8 raw[V], add[V];
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = ((c * W + in_row) * 32 + lane) * 8;
      if (live && col < D) {
        raw[c] = *reinterpret_cast<const bf16x8*>(in + col);
        if (delta) add[c] = *reinterpret_cast<const bf16x8*>(in + static_cast<size_t>(R) * D + col);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars.empty[s]);
    float part[V];
#pragma unroll
    for (int c = 0; c < V; ++c) part[c] = 0.f;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = ((c * W + in_row) * 32 + lane) * 8;
      if (live && col < D) {
        float v[8];
        unpack8(raw[c], v);
        if (delta) {
          float d[8];
          unpack8(add[c], d);
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] += d[i];
          // the sum is rounded to bf16 once; the norm sees the rounded value, like the unfused path
          raw[c] = pack8(v);
          *reinterpret_cast<bf16x8*>(sum_out + base + col) = raw[c];
          unpack8(raw[c], v);
        }
        float& ss = part[W == 8 ? 0 : c];
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
      }
    }
    const float total = norm_row_sum<W, V>(part, scratch[count & 1], slot, in_row, lane);
    const float r = rsqrtf(total / D + eps);
    if (live && in_row == 0 && lane == 0) rstd[row] = r;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = ((c * W + in_row) * 32 + lane) * 8;
      if (live && col < D) {
        float v[8], o[8];
        unpack8(raw[c], v);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = v[i] * r * wv[c][i];
        *reinterpret_cast<bf16x8*>(y + base + col) = pack8(o);
      }
    }
  }
}

// The same for few rows, one CTA per row (grid-stride), straight from global memory: a ring has nothing to read ahead where
// a CTA has one block of rows (200 x 512: 1.8 us here, 2.6 there).  CH = 8-element vectors per thread.  Same sums, same bits.
template <int CH>
__global__ void __launch_bounds__(NORM_THREADS) rmsnorm_fwd_row_kernel(const __nv_bfloat16* __restrict__ x,
                                                                  const __nv_bfloat16* __restrict__ delta,
                                                                  const float* __restrict__ w,
                                                                  __nv_bfloat16* __restrict__ sum_out,
                                                                  __nv_bfloat16* __restrict__ y,
                                                                  float* __restrict__ rstd, int rows, int D, float eps) {
  chain_begin();
  __shared__ float scratch[NORM_THREADS / 32];
  float wv[CH][8];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int col = (c * NORM_THREADS + threadIdx.x) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) wv[c][i] = col < D ? w[col + i] : 0.f;
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = static_cast<size_t>(row) * D;
    bf16x8 raw[CH];
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int col = (c * NORM_THREADS + threadIdx.x) * 8;
      if (col < D) {
        raw[c] = *reinterpret_cast<const bf16x8*>(x + base + col);
        float v[8];
        unpack8(raw[c], v);
        if (delta) {
          float d[8];
          unpack8(*reinterpret_cast<const bf16x8*>(delta + base + col), d);
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] += d[i];
          // the sum is rounded to bf16 once; the norm sees the rounded value, like the unfused path
          raw[c] = pack8(v);
          *reinterpret_cast<bf16x8*>(sum_out + base + col) = raw[c];
          unpack8(raw[c], v);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
      }
    }
    const float total = block_sum<NORM_THREADS>(ss, scratch);
    const float r = rsqrtf(total / D + eps);
    if (threadIdx.x == 0) rstd[row] = r;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int col = (c * NORM_THREADS + threadIdx.x) * 8;
      if (col < D) {
        float v[8], o[8];
        unpack8(raw[c], v);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = v[i] * r * wv[c][i];
        *reinterpret_cast<bf16x8*>(y + base + col) = pack8(o);
      }
    }
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) [+ residual]; dw partial per CTA.  RING 0: no CTA has more than one block of rows,
// which its warps read straight from global memory (us with the column sum: 1 x 512 4.0 -> 3.7, 300 x 2048 7.5 -> 6.7).
template <int W, int V, int RING>
__global__ void __launch_bounds__(NORM_THREADS + 32, V == 2 ? 2 : 1)
    rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                       const float* __restrict__ w, const float* __restrict__ rstd,
                       const __nv_bfloat16* residual, __nv_bfloat16* dx, float* __restrict__ dw_partial,
                       int* __restrict__ status, int rows, int D, int ring_stages) {
  chain_begin();
  constexpr int R = 8 / W;
  extern __shared__ __align__(128) uint8_t norm_ring[];
  __shared__ NormBars bars;
  __shared__ float scratch[2][R][8];
  if (RING) norm_init(bars);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool worker = warp < NORM_THREADS / 32;
  const int slot = warp / W, in_row = warp % W;
  float dw_acc[V][8];
  if (!worker) {
    const __nv_bfloat16* const src[3] = {dy, x, residual};
    norm_producer<R, 3>(src, norm_ring, ring_stages, bars, status, rows, D);
    __syncwarp();
  } else {
    float wv[V][8];
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = ((c * W + in_row) * 32 + lane) * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        dw_acc[c][i] = 0.f;
        wv[c][i] = col < D ? w[col + i] : 0.f;
      }
    }
    const int blocks = (rows + R - 1) / R;
    int count = 0;
    bool here = true;
    float next_r = static_cast<int>(blockIdx.x) * R + slot < rows ? rstd[blockIdx.x * R + slot] : 0.f;
    for (int block = blockIdx.x; block < blocks; block += gridDim.x, ++count) {
      const int s = RING ? count % ring_stages : 0;
      const int row = block * R + slot, after = row + static_cast<int>(gridDim.x) * R;
      const bool live = row < rows;
      const float r = next_r;
      if (after < rows) next_r = rstd[after];
      const __nv_bfloat16* in = reinterpret_cast<const __nv_bfloat16*>(norm_ring) + (static_cast<size_t>(s) * 3 * R + slot) * D;
      const size_t base = static_cast<size_t>(row) * D;
      if (RING) here = norm_arrived(here, bars.full[s], (count / ring_stages) & 1, status);
      bf16x8 a[V], b[V], res[V];
#pragma unroll
      for (int c = 0; c < V; ++c) {
        const int col = ((c * W + in_row) * 32 + lane) * 8;
        if (live && col < D) {
          a[c] = *reinterpret_cast<const bf16x8*>(RING ? in + col : dy + base + col);
          b[c] = *reinterpret_cast<const bf16x8*>(RING ? in + static_cast<size_t>(R) * D + col : x + base + col);
          if (residual)
            res[c] = *reinterpret_cast<const bf16x8*>(RING ? in + static_cast<size_t>(2 * R) * D + col : residual + base + col);
        }
      }
      __syncwarp();
      if (RING && lane == 0) mbar_arrive(&bars.empty[s]);
      float part[V];
#pragma unroll
      for (int c = 0; c < V; ++c) part[c] = 0.f;
#pragma unroll
      for (int c = 0; c < V; ++c) {
        const int col = ((c * W + in_row) * 32 + lane) * 8;
        if (live && col < D) {
          float dyv[8], xv[8];
          unpack8(a[c], dyv);
          unpack8(b[c], xv);
          float& dot = part[W == 8 ? 0 : c];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float xh = xv[i] * r;
            dw_acc[c][i] += dyv[i] * xh;
            dot += dyv[i] * wv[c][i] * xh;
          }
        }
      }
      const float mean = norm_row_sum<W, V>(part, scratch[count & 1], slot, in_row, lane) / D;
#pragma unroll
      for (int c = 0; c < V; ++c) {
        const int col = ((c * W + in_row) * 32 + lane) * 8;
        if (live && col < D) {
          float dyv[8], xv[8], o[8];
          unpack8(a[c], dyv);
          unpack8(b[c], xv);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = r * (dyv[i] * wv[c][i] - xv[i] * r * mean);
          if (residual) {
            float add[8];
            unpack8(res[c], add);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] += add[i];
          }
          *reinterpret_cast<bf16x8*>(dx + base + col) = pack8(o);
        }
      }
    }
  }
  // the rows that the CTA worked on at the same time are added up in the ring, whose copies have all been taken
  float* const sums = reinterpret_cast<float*>(norm_ring);
  __syncthreads();
  if (W < 8) {
    if (worker) {
#pragma unroll
      for (int c = 0; c < V; ++c) {
        const int col = ((c * W + in_row) * 32 + lane) * 8;
        if (col < D) {
          float4* const dst = reinterpret_cast<float4*>(sums + static_cast<size_t>(slot) * D + col);
          dst[0] = make_float4(dw_acc[c][0], dw_acc[c][1], dw_acc[c][2], dw_acc[c][3]);
          dst[1] = make_float4(dw_acc[c][4], dw_acc[c][5], dw_acc[c][6], dw_acc[c][7]);
        }
      }
    }
    __syncthreads();
    for (int col = threadIdx.x; col < D; col += blockDim.x) {
      float total = 0.f;
#pragma unroll
      for (int k = 0; k < R; ++k) total += sums[static_cast<size_t>(k) * D + col];
      dw_partial[static_cast<size_t>(blockIdx.x) * D + col] = total;
    }
  } else if (worker) {
#pragma unroll
    for (int c = 0; c < V; ++c) {
      const int col = ((c * W + in_row) * 32 + lane) * 8;
      if (col < D) {
        float4* const dst = reinterpret_cast<float4*>(dw_partial + static_cast<size_t>(blockIdx.x) * D + col);
        dst[0] = make_float4(dw_acc[c][0], dw_acc[c][1], dw_acc[c][2], dw_acc[c][3]);
        dst[1] = make_float4(dw_acc[c][4], dw_acc[c][5], dw_acc[c][6], dw_acc[c][7]);
      }
    }
  }
}

// out[col] = sum over parts of partial[part][col].  One CTA per 32 columns: lane = column (coalesced 128-byte reads), the
// 32 warps take every 32nd part (eight warps in four chains each were 7.6 us at 296 parts of 512 columns, this 2.5),
// shared memory adds the 32 partial sums.  Eight warps for up to eight parts: the same sums without the warps that add zeros.
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) column_sum_kernel(const float* __restrict__ partial, float* __restrict__ out,
                                                         int parts, int D) {
  chain_begin();
  __shared__ float acc[WARPS][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (col < D) {
#pragma unroll 10
    for (int p = warp; p < parts; p += WARPS) s += partial[static_cast<size_t>(p) * D + col];
  }
  acc[warp][lane] = s;
  __syncthreads();
#pragma unroll
  for (int c = warp; c < 32; c += WARPS) {    // transposed: warp = column, lane = part
    s = warp_sum(lane < WARPS ? acc[lane][c] : 0.f);
    if (lane == 0 && blockIdx.x * 32 + c < D) out[blockIdx.x * 32 + c] = s;
  }
}

// ------------------------------------------------------------------ router softmax / top-2
constexpr int ROUTER_MAX_E = 64;

// Softmax over E <= MAXE experts and the renormalised weights of the two largest, one thread per row.
template <int MAXE>
__device__ __forceinline__ void top2_row(const float* __restrict__ logits, float* __restrict__ weights,
                                         long long* __restrict__ idx, float* __restrict__ probs, int E) {
  float p[MAXE];
  float mx = -INFINITY;
  for (int e = 0; e < E; ++e) {
    p[e] = logits[e];
    mx = fmaxf(mx, p[e]);
  }
  float sum = 0.f;
  for (int e = 0; e < E; ++e) {
    p[e] = __expf(p[e] - mx);
    sum += p[e];
  }
  const float inv = 1.f / sum;
  int a = 0, b = -1;
  float pa = -1.f, pb = -1.f;
  for (int e = 0; e < E; ++e) {
    p[e] *= inv;
    probs[e] = p[e];
    if (p[e] > pa) {           // strict: ties keep the lower index first, like topk
      pb = pa; b = a;
      pa = p[e]; a = e;
    } else if (p[e] > pb) {
      pb = p[e]; b = e;
    }
  }
  if (b < 0) {                 // only reachable with non-finite logits: keep the indices valid
    b = a == 0 ? 1 : 0;
    pb = p[b];
  }
  const float s = pa + pb;
  weights[0] = pa / s;
  weights[1] = pb / s;
  idx[0] = a;
  idx[1] = b;
}

__global__ void router_top2_fwd_kernel(const float* __restrict__ logits, float* __restrict__ weights,
                                       long long* __restrict__ idx, float* __restrict__ probs, int T, int E) {
  chain_begin();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  const size_t row = static_cast<size_t>(t) * E;
  top2_row<ROUTER_MAX_E>(logits + row, weights + 2 * static_cast<size_t>(t), idx + 2 * static_cast<size_t>(t), probs + row, E);
}

// ------------------------------------------------------------------ skinny linear (router: N <= 16 outputs)
constexpr int SKINNY_MAX_N = 16;

// The three kernels are bound by reading or writing the activations once.  A warp works on four tokens at a time, so
// that an unpacked weight serves four of them: with one token per warp the shared-memory reads and conversions of the
// weights were the limit (5003 x 4096, 8 outputs: nt 56 -> 34 us, nn 51 -> 33 us; 16384 tokens: 149 -> 66, 127 -> 64).
constexpr int SKINNY_TOKENS = 4;

__device__ __forceinline__ void skinny_stage(__nv_bfloat16* ws, const __nv_bfloat16* __restrict__ w, int count) {
  for (int i = threadIdx.x * 8; i < count; i += blockDim.x * 8)
    *reinterpret_cast<bf16x8*>(ws + i) = *reinterpret_cast<const bf16x8*>(w + i);
  __syncthreads();
}

// Sums 32 values over the warp: lane i returns the sum of v[i] over all lanes (31 shuffles instead of 160).
__device__ __forceinline__ float warp_sum_scatter(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float keep = upper ? v[i + o] : v[i], send = upper ? v[i] : v[i + o];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// logits[t, n] = sum_k x[t,k] w[n,k]; weights in shared memory.  NN: N rounded up to 8 or 16.  With TOP2 the router's
// softmax and choice follow in the same launch (four lanes, a token each) and the product itself is not stored.
template <int NN, bool TOP2>
__global__ void __launch_bounds__(256) skinny_nt_kernel(const __nv_bfloat16* __restrict__ x,
                                                        const __nv_bfloat16* __restrict__ w, float* __restrict__ out,
                                                        float* __restrict__ weights, long long* __restrict__ idx,
                                                        float* __restrict__ probs, int T, int N, int K) {
  chain_begin();
  extern __shared__ __nv_bfloat16 ws[];
  __shared__ float chosen[TOP2 ? 8 : 1][SKINNY_TOKENS][NN];
  skinny_stage(ws, w, N * K);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t0 = (blockIdx.x * 8 + warp) * SKINNY_TOKENS; t0 < T; t0 += gridDim.x * 8 * SKINNY_TOKENS) {
    float acc[NN / 8][SKINNY_TOKENS * 8];
#pragma unroll
    for (int h = 0; h < NN / 8; ++h)
#pragma unroll
      for (int i = 0; i < SKINNY_TOKENS * 8; ++i) acc[h][i] = 0.f;
    const __nv_bfloat16* row[SKINNY_TOKENS];
#pragma unroll
    for (int j = 0; j < SKINNY_TOKENS; ++j) row[j] = x + static_cast<size_t>(min(t0 + j, T - 1)) * K;
    bf16x8 next[SKINNY_TOKENS];
    if (lane * 8 < K) {
#pragma unroll
      for (int j = 0; j < SKINNY_TOKENS; ++j) next[j] = *reinterpret_cast<const bf16x8*>(row[j] + lane * 8);
    }
    for (int k = lane * 8; k < K; k += 256) {
      float xv[SKINNY_TOKENS][8];
#pragma unroll
      for (int j = 0; j < SKINNY_TOKENS; ++j) unpack8(next[j], xv[j]);
      if (k + 256 < K) {
#pragma unroll
        for (int j = 0; j < SKINNY_TOKENS; ++j) next[j] = *reinterpret_cast<const bf16x8*>(row[j] + k + 256);
      }
#pragma unroll
      for (int n = 0; n < NN; ++n) {
        if (n < N) {
          float wv[8];
          unpack8(*reinterpret_cast<const bf16x8*>(ws + n * K + k), wv);
#pragma unroll
          for (int j = 0; j < SKINNY_TOKENS; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[n / 8][j * 8 + n % 8] += xv[j][i] * wv[i];
        }
      }
    }
#pragma unroll
    for (int h = 0; h < NN / 8; ++h) {
      const float sum = warp_sum_scatter(acc[h], lane);
      const int t = t0 + lane / 8, n = h * 8 + lane % 8;
      if (!TOP2 && t < T && n < N) out[static_cast<size_t>(t) * N + n] = sum;
      if (TOP2) chosen[warp][lane / 8][n] = sum;
    }
    if (TOP2) {
      __syncwarp();
      const size_t t = t0 + lane;
      if (lane < SKINNY_TOKENS && t < T) top2_row<NN>(chosen[warp][lane], weights + 2 * t, idx + 2 * t, probs + t * N, N);
      __syncwarp();
    }
  }
}

// dx[t,k] = sum_n dy[t,n] w[n,k]  (bf16 out)
template <int NN>
__global__ void __launch_bounds__(256) skinny_nn_kernel(const float* __restrict__ dy,
                                                        const __nv_bfloat16* __restrict__ w,
                                                        __nv_bfloat16* __restrict__ dx, int T, int N, int K) {
  chain_begin();
  extern __shared__ __nv_bfloat16 ws[];
  skinny_stage(ws, w, N * K);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t0 = (blockIdx.x * 8 + warp) * SKINNY_TOKENS; t0 < T; t0 += gridDim.x * 8 * SKINNY_TOKENS) {
    float d[SKINNY_TOKENS][NN];
#pragma unroll
    for (int j = 0; j < SKINNY_TOKENS; ++j)
#pragma unroll
      for (int n = 0; n < NN; ++n) d[j][n] = n < N ? dy[static_cast<size_t>(min(t0 + j, T - 1)) * N + n] : 0.f;
    for (int k = lane * 8; k < K; k += 256) {
      float o[SKINNY_TOKENS][8];
#pragma unroll
      for (int j = 0; j < SKINNY_TOKENS; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) o[j][i] = 0.f;
#pragma unroll
      for (int n = 0; n < NN; ++n) {
        if (n < N) {
          float wv[8];
          unpack8(*reinterpret_cast<const bf16x8*>(ws + n * K + k), wv);
#pragma unroll
          for (int j = 0; j < SKINNY_TOKENS; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) o[j][i] += d[j][n] * wv[i];
        }
      }
#pragma unroll
      for (int j = 0; j < SKINNY_TOKENS; ++j)
        if (t0 + j < T) *reinterpret_cast<bf16x8*>(dx + static_cast<size_t>(t0 + j) * K + k) = pack8(o[j]);
    }
  }
}

// dw[n,k] += sum_t dy[t,n] x[t,k].  A CTA owns 256 columns and a range of tokens; its eight warps take every eighth
// token, shared memory adds their sums, and one atomic per (n, column) and CTA goes to dw.  Wide CTAs (2048 columns, 32
// tokens) spent their time in the atomics, one per 32 tokens: 113 -> 35 us at 5003 x 4096, 8 outputs.
template <int NN>
__global__ void __launch_bounds__(256) skinny_tn_kernel(const float* __restrict__ dy,
                                                        const __nv_bfloat16* __restrict__ x, float* __restrict__ dw,
                                                        int T, int N, int K, int tokens_per_cta) {
  chain_begin();
  __shared__ float sums[8][8][32 + 1];       // [warp][column of the lane][lane], one output at a time
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = blockIdx.x * 256 + lane * 8;
  const int t0 = blockIdx.y * tokens_per_cta;
  const int t1 = min(T, t0 + tokens_per_cta);
  float acc[NN][8];
#pragma unroll
  for (int n = 0; n < NN; ++n)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[n][i] = 0.f;
  if (k < K) {
#pragma unroll 4
    for (int t = t0 + warp; t < t1; t += 8) {
      float xv[8];
      unpack8(*reinterpret_cast<const bf16x8*>(x + static_cast<size_t>(t) * K + k), xv);
#pragma unroll
      for (int n = 0; n < NN; ++n) {
        if (n < N) {
          const float d = dy[static_cast<size_t>(t) * N + n];
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[n][i] += d * xv[i];
        }
      }
    }
  }
  const int col = threadIdx.x;               // column of the CTA that this thread adds up
#pragma unroll
  for (int n = 0; n < NN; ++n) {
    if (n < N) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 8; ++i) sums[warp][i][lane] = acc[n][i];
      __syncthreads();
      float total = 0.f;
#pragma unroll
      for (int v = 0; v < 8; ++v) total += sums[v][col & 7][col >> 3];
      if (blockIdx.x * 256 + col < K) atomicAdd(dw + static_cast<size_t>(n) * K + blockIdx.x * 256 + col, total);
    }
  }
}

// ------------------------------------------------------------------ router backward
__global__ void router_top2_bwd_kernel(const float* __restrict__ dweights, const float* __restrict__ probs,
                                       const long long* __restrict__ idx, const float* __restrict__ weights,
                                       float* __restrict__ dlogits, int T, int E) {
  chain_begin();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  const int a = static_cast<int>(idx[2 * t]), b = static_cast<int>(idx[2 * t + 1]);
  const float wa = weights[2 * t], wb = weights[2 * t + 1];
  const float da = dweights[2 * t], db = dweights[2 * t + 1];
  const float pa = probs[static_cast<size_t>(t) * E + a], pb = probs[static_cast<size_t>(t) * E + b];
  const float s = pa + pb;
  const float inner = da * wa + db * wb;
  const float dpa = (da - inner) / s, dpb = (db - inner) / s;
  const float dot = dpa * pa + dpb * pb;
  for (int e = 0; e < E; ++e) {
    const float p = probs[static_cast<size_t>(t) * E + e];
    const float dp = e == a ? dpa : (e == b ? dpb : 0.f);
    dlogits[static_cast<size_t>(t) * E + e] = p * (dp - dot);
  }
}

// ------------------------------------------------------------------ SwiGLU backward
// dgu[r, 0:F] = dh * u * silu'(g); dgu[r, F:2F] = dh * silu(g); h = silu(g) * u
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dh, const __nv_bfloat16* __restrict__ gate,
                                  const __nv_bfloat16* __restrict__ up, __nv_bfloat16* __restrict__ dgu,
                                  __nv_bfloat16* __restrict__ h, const int* __restrict__ live_rows, int rows, int F) {
  chain_begin();
  const int limit = live_rows ? min(rows, *live_rows) : rows;
  const size_t per_row = F / 8;
  const size_t total = static_cast<size_t>(limit) * per_row;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t row = i / per_row;
    const size_t col = (i - row * per_row) * 8;
    float d[8], g[8], u[8], og[8], ou[8], oh[8];
    unpack8(*reinterpret_cast<const bf16x8*>(dh + row * F + col), d);
    unpack8(*reinterpret_cast<const bf16x8*>(gate + row * F + col), g);
    unpack8(*reinterpret_cast<const bf16x8*>(up + row * F + col), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sig = 1.f / (1.f + __expf(-g[j]));
      const float sl = g[j] * sig;
      og[j] = d[j] * u[j] * sig * (1.f + g[j] * (1.f - sig));
      ou[j] = d[j] * sl;
      oh[j] = sl * u[j];
    }
    *reinterpret_cast<bf16x8*>(dgu + row * 2 * F + col) = pack8(og);
    *reinterpret_cast<bf16x8*>(dgu + row * 2 * F + F + col) = pack8(ou);
    if (h) *reinterpret_cast<bf16x8*>(h + row * F + col) = pack8(oh);
  }
}

// ------------------------------------------------------------------ cross entropy (in place)
// logits[t,:] <- (softmax(logits[t,:]) - onehot(target)) * scale ; loss += (lse - logit[target]) * scale
constexpr int CE_THREADS = 512;

// A CTA's part of the loss, from one thread.  ``wide``: the sum is a double, so that it does not depend on the order of the
// CTAs as far as fp32 can tell (hundreds of fp32 additions in the order of their arrival are off by 1e-7 from run to run).
__device__ __forceinline__ void add_loss(void* loss, int wide, double value) {
  if (wide) atomicAdd(static_cast<double*>(loss), value);
  else atomicAdd(static_cast<float*>(loss), static_cast<float>(value));
}
__global__ void __launch_bounds__(CE_THREADS) cross_entropy_kernel(__nv_bfloat16* __restrict__ logits,
                                                                  const long long* __restrict__ targets,
                                                                  void* __restrict__ loss, int wide, int T, int V,
                                                                  float scale) {
  chain_begin();
  __shared__ float scratch[CE_THREADS / 32];
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    __nv_bfloat16* row = logits + static_cast<size_t>(t) * V;
    float mx = -INFINITY;
    for (int c = threadIdx.x * 8; c < V; c += CE_THREADS * 8) {
      float v[8];
      unpack8(*reinterpret_cast<const bf16x8*>(row + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) mx = fmaxf(mx, v[i]);
    }
    mx = block_max<CE_THREADS>(mx, scratch);
    float sum = 0.f;
    for (int c = threadIdx.x * 8; c < V; c += CE_THREADS * 8) {
      float v[8];
      unpack8(*reinterpret_cast<const bf16x8*>(row + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) sum += __expf(v[i] - mx);
    }
    sum = block_sum<CE_THREADS>(sum, scratch);
    const float inv = 1.f / sum;
    const int target = static_cast<int>(targets[t]);
    if (threadIdx.x == 0) {
      const float picked = __bfloat162float(row[target]);
      add_loss(loss, wide, (logf(sum) + mx - picked) * scale);
    }
    __syncthreads();
    for (int c = threadIdx.x * 8; c < V; c += CE_THREADS * 8) {
      float v[8];
      unpack8(*reinterpret_cast<const bf16x8*>(row + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] = __expf(v[i] - mx) * inv;
        if (c + i == target) v[i] -= 1.f;
        v[i] *= scale;
      }
      *reinterpret_cast<bf16x8*>(row + c) = pack8(v);
    }
  }
}

// The same with one read and one write of the logits instead of three reads and one write.  ``loss_scale`` weighs the
// row's loss in ``loss`` (1/T for a mean over T tokens), ``grad_scale`` multiplies the gradient written back (1/T times
// whatever the caller back-propagates into the loss).  Two CTAs per SM; the target's entry is looked for once per vector
// and its logit read beside the row (what is done per element counts as much as the traffic).
constexpr int CE_REG_CHUNKS = 8;

// Rows up to 16384 entries (CHUNKS 2 or 4): each exponential is formed once and kept in fp32, and as soon as a vector of
// the row has been used the same vector of the CTA's next row is requested.  4096 x 2048: 45 -> 21 us, 4096 x 16000:
// 103 -> 70 us (exponentials formed twice, loads exposed before).
template <int CHUNKS>
__global__ void __launch_bounds__(CE_THREADS, 2)
    cross_entropy_reg_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets,
                             void* __restrict__ loss, int wide, int T, int V, float loss_scale, float grad_scale) {
  chain_begin();
  __shared__ float scratch[CE_THREADS / 32];
  double local_loss = 0.;
  bf16x8 raw[CHUNKS];
  if (blockIdx.x < T) {
    const __nv_bfloat16* row = logits + static_cast<size_t>(blockIdx.x) * V;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = (k * CE_THREADS + threadIdx.x) * 8;
      if (c < V) raw[k] = *reinterpret_cast<const bf16x8*>(row + c);
    }
  }
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    __nv_bfloat16* row = logits + static_cast<size_t>(t) * V;
    const __nv_bfloat16* next = row + static_cast<size_t>(gridDim.x) * V;
    const bool more = t + static_cast<int>(gridDim.x) < T;
    const int target = static_cast<int>(targets[t]);
    const bool valid = target >= 0 && target < V;
    const float picked = valid && threadIdx.x == 0 ? __bfloat162float(row[target]) : 0.f;
    float mx = -INFINITY;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = (k * CE_THREADS + threadIdx.x) * 8;
      if (c < V) {
        float v[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, v[i]);
      }
    }
    mx = block_max<CE_THREADS>(mx, scratch);
    float e[CHUNKS][8], sum = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = (k * CE_THREADS + threadIdx.x) * 8;
      if (c < V) {
        unpack8(raw[k], e[k]);
        if (more) raw[k] = *reinterpret_cast<const bf16x8*>(next + c);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          e[k][i] = __expf(e[k][i] - mx);
          sum += e[k][i];
        }
      }
    }
    sum = block_sum<CE_THREADS>(sum, scratch);
    const float inv = 1.f / sum;
    if (valid && threadIdx.x == 0) local_loss += (logf(sum) + mx - picked) * loss_scale;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = (k * CE_THREADS + threadIdx.x) * 8;
      if (c < V) {
#pragma unroll
        for (int i = 0; i < 8; ++i) e[k][i] *= inv;
        if (c <= target && target < c + 8) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (c + i == target) e[k][i] -= 1.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) e[k][i] *= grad_scale;
        *reinterpret_cast<bf16x8*>(row + c) = pack8(e[k]);
      }
    }
  }
  if (threadIdx.x == 0 && local_loss != 0.) add_loss(loss, wide, local_loss);   // one atomic per CTA
}

// Rows up to 32768 entries: the registers of two CTAs hold the packed rows, not their exponentials in fp32 (formed twice;
// one CTA per SM that keeps them took 215 us where two that do not took 165 at 4096 x 32000).  The CTA's next row arrives
// in shared memory by one bulk copy while the present one is worked on: 165 -> 124 us, 16384 rows 628 -> 467 us.
__global__ void __launch_bounds__(CE_THREADS, 2)
    cross_entropy_bulk_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets,
                              void* __restrict__ loss, int wide, int* __restrict__ status, int T, int V,
                              float loss_scale, float grad_scale) {
  chain_begin();
  extern __shared__ __align__(128) uint8_t ce_row[];
  __shared__ float scratch[CE_THREADS / 32];
  __shared__ uint64_t arrived;
  const uint32_t bytes = static_cast<uint32_t>(V) * 2;
  if (threadIdx.x == 0) {
    mbar_init(&arrived, 1);
    mbar_fence_init();
    if (blockIdx.x < T) {
      mbar_expect_tx(&arrived, bytes);
      bulk_load(ce_row, logits + static_cast<size_t>(blockIdx.x) * V, &arrived, bytes);
    }
  }
  __syncthreads();
  double local_loss = 0.;
  uint32_t phase = 0;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    __nv_bfloat16* row = logits + static_cast<size_t>(t) * V;
    const int target = static_cast<int>(targets[t]);
    const bool valid = target >= 0 && target < V;
    const bool here = mbar_wait(&arrived, phase);
    phase ^= 1;
    if (__syncthreads_or(!here)) {            // a copy did not arrive in time: report and leave, all threads alike
      if (threadIdx.x == 0) {
        atomicExch(status, 5);
        mbar_wait(&arrived, phase ^ 1);       // it may still land in this CTA's memory: one more limit's time
      }
      break;
    }
    const float picked =
        valid && threadIdx.x == 0 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ce_row)[target]) : 0.f;
    bf16x8 raw[CE_REG_CHUNKS];
    float mx = -INFINITY;
#pragma unroll
    for (int k = 0; k < CE_REG_CHUNKS; ++k) {
      const int c = (k * CE_THREADS + threadIdx.x) * 8;
      if (c < V) {
        raw[k] = *reinterpret_cast<const bf16x8*>(ce_row + c * 2);
        float v[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, v[i]);
      }
    }
    mx = block_max<CE_THREADS>(mx, scratch);
    // every thread has taken its part of the row: the next one may overwrite it
    if (threadIdx.x == 0 && t + static_cast<int>(gridDim.x) < T) {
      fence_async_shared();
      mbar_expect_tx(&arrived, bytes);
      bulk_load(ce_row, row + static_cast<size_t>(gridDim.x) * V, &arrived, bytes);
    }
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < CE_REG_CHUNKS; ++k) {
      const int c = (k * CE_THREADS + threadIdx.x) * 8;
      if (c < V) {
        float v[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += __expf(v[i] - mx);
      }
    }
    sum = block_sum<CE_THREADS>(sum, scratch);
    const float inv = 1.f / sum;
    if (valid && threadIdx.x == 0) local_loss += (logf(sum) + mx - picked) * loss_scale;
#pragma unroll
    for (int k = 0; k < CE_REG_CHUNKS; ++k) {
      const int c = (k * CE_THREADS + threadIdx.x) * 8;
      if (c < V) {
        float v[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __expf(v[i] - mx) * inv;
        if (c <= target && target < c + 8) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (c + i == target) v[i] -= 1.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] *= grad_scale;
        *reinterpret_cast<bf16x8*>(row + c) = pack8(v);
      }
    }
  }
  if (threadIdx.x == 0 && local_loss != 0.) add_loss(loss, wide, local_loss);   // one atomic per CTA
}

__global__ void scale_bf16_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ factor, size_t n8) {
  chain_begin();
  const float f = *factor;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n8;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    float v[8];
    unpack8(reinterpret_cast<const bf16x8*>(x)[i], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= f;
    reinterpret_cast<bf16x8*>(x)[i] = pack8(v);
  }
}

// ------------------------------------------------------------------ AdamW
template <typename T>
__device__ __forceinline__ float ldf(const T* p, size_t i);
template <>
__device__ __forceinline__ float ldf<float>(const float* p, size_t i) { return p[i]; }
template <>
__device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, size_t i) { return __bfloat162float(p[i]); }
template <typename T>
__device__ __forceinline__ void stf(T* p, size_t i, float v);
template <>
__device__ __forceinline__ void stf<float>(float* p, size_t i, float v) { p[i] = v; }
template <>
__device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, size_t i, float v) { p[i] = __float2bfloat16_rn(v); }

template <typename T>
__device__ __forceinline__ void ld8(const T* p, float (&f)[8]);
template <>
__device__ __forceinline__ void ld8<float>(const float* p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <>
__device__ __forceinline__ void ld8<__nv_bfloat16>(const __nv_bfloat16* p, float (&f)[8]) {
  unpack8(*reinterpret_cast<const bf16x8*>(p), f);
}
template <typename T>
__device__ __forceinline__ void st8(T* p, const float (&f)[8]);
template <>
__device__ __forceinline__ void st8<float>(float* p, const float (&f)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
template <>
__device__ __forceinline__ void st8<__nv_bfloat16>(__nv_bfloat16* p, const float (&f)[8]) {
  *reinterpret_cast<bf16x8*>(p) = pack8(f);
}

// Up to ADAMW_MAX tensors of the same types per launch; the table travels as a kernel argument.  Tensors are cut into
// blocks that the CTAs take in turn, so that gains of a few thousand elements share a launch with expert stacks (one
// launch per tensor left the chip idle between them).  Blocks of ADAMW_CHUNK elements where they fill the launch's 16
// CTAs per SM; below that one vector per thread, or a launch is as long as a CTA's four turns (100003 fp32 elements 6.3
// -> 3.0 us, 2^20 bf16 6.3 -> 4.1, 10^7 fp32 48.4 -> 45.1).  Bound by memory traffic.
constexpr int ADAMW_MAX = 48;
constexpr int ADAMW_CHUNK = 8192, ADAMW_SMALL_CHUNK = 2048;
struct AdamwTensor {
  void* p;
  const void* g;
  void* m;
  void* v;
  __nv_bfloat16* p_bf16;     // optional copy of the new p
  long long n;
};
struct AdamwTable {
  AdamwTensor t[ADAMW_MAX];
  int first_chunk[ADAMW_MAX + 1];
  int count;
  int chunk;                 // elements per block
};

// p <- p(1 - lr*wd); m, v moments; p <- p - a_t m/(sqrt(v)+eps).  Optional bf16 copy of the new p.
// Eight elements per thread as 16/32-byte vectors; the last n % 8 elements go one by one.
template <typename P, typename G, typename S>
__global__ void __launch_bounds__(256) adamw_kernel(const __grid_constant__ AdamwTable table, float lr, float beta1,
                                                    float beta2, float eps, float wd, float a_t, float grad_scale) {
  chain_begin();
  const float decay = 1.f - lr * wd;
  int which = 0;
  for (int chunk = blockIdx.x; chunk < table.first_chunk[table.count]; chunk += gridDim.x) {
    while (chunk >= table.first_chunk[which + 1]) ++which;
    const AdamwTensor& t = table.t[which];
    P* __restrict__ p = static_cast<P*>(t.p);
    const G* __restrict__ g = static_cast<const G*>(t.g);
    S* __restrict__ m = static_cast<S*>(t.m);
    S* __restrict__ v = static_cast<S*>(t.v);
    const size_t begin = static_cast<size_t>(chunk - table.first_chunk[which]) * table.chunk;
    const size_t n = static_cast<size_t>(t.n);
    const size_t end = begin + table.chunk < n ? begin + table.chunk : n;
    for (size_t o = begin + threadIdx.x * 8; o + 8 <= end; o += 256 * 8) {
      float pv[8], gv[8], mv[8], vv[8];
      ld8(p + o, pv);
      ld8(g + o, gv);
      ld8(m + o, mv);
      ld8(v + o, vv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float gj = gv[j] * grad_scale;
        mv[j] = beta1 * mv[j] + (1.f - beta1) * gj;
        vv[j] = beta2 * vv[j] + (1.f - beta2) * gj * gj;
        pv[j] = pv[j] * decay - a_t * mv[j] / (sqrtf(vv[j]) + eps);
      }
      st8(p + o, pv);
      st8(m + o, mv);
      st8(v + o, vv);
      if (t.p_bf16) st8(t.p_bf16 + o, pv);
    }
    for (size_t i = begin + (end - begin) / 8 * 8 + threadIdx.x; i < end; i += 256) {   // only behind the last vector
      const float gj = ldf(g, i) * grad_scale;
      const float mj = beta1 * ldf(m, i) + (1.f - beta1) * gj;
      const float vj = beta2 * ldf(v, i) + (1.f - beta2) * gj * gj;
      const float pj = ldf(p, i) * decay - a_t * mj / (sqrtf(vj) + eps);
      stf(p, i, pj);
      stf(m, i, mj);
      stf(v, i, vj);
      if (t.p_bf16) t.p_bf16[i] = __float2bfloat16_rn(pj);
    }
  }
}

// Zeros into up to ZERO_MAX buffers in one launch: a CTA per 8 KiB, 32 bytes per thread, no loop.  Bound by the writes to
// memory, which arrive in order this way: 5.9 GB in 783 us, 7.5 TB/s (a copy measures 6.45).  Eight persistent CTAs per SM
// that take 64 KiB in turn, with 16-byte stores, need 978, with 32-byte stores 962; bulk copies of a zeroed buffer 927;
// cudaMemset 805.
constexpr int ZERO_MAX = 64;
constexpr int ZERO_CHUNK = 8192;
struct ZeroTable {
  uint8_t* p[ZERO_MAX];
  long long bytes[ZERO_MAX];
  int first_chunk[ZERO_MAX + 1];
  int count;
};
__global__ void __launch_bounds__(256) zero_kernel(const __grid_constant__ ZeroTable table) {
  chain_begin();
  const int chunk = blockIdx.x;
  int which = 0, end = table.count;          // the last buffer that starts at or before this chunk
  while (end - which > 1) {
    const int mid = (which + end) / 2;
    if (table.first_chunk[mid] <= chunk) which = mid;
    else end = mid;
  }
  const size_t at = static_cast<size_t>(chunk - table.first_chunk[which]) * ZERO_CHUNK + threadIdx.x * 32;
  const size_t bytes = static_cast<size_t>(table.bytes[which]);
  uint8_t* const dst = table.p[which] + at;
  if (at + 32 <= bytes) {
    if ((reinterpret_cast<uintptr_t>(dst) & 31) == 0) {
      asm volatile("st.global.v8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"l"(dst), "r"(0) : "memory");
    } else {
      reinterpret_cast<uint4*>(dst)[0] = make_uint4(0, 0, 0, 0);
      reinterpret_cast<uint4*>(dst)[1] = make_uint4(0, 0, 0, 0);
    }
  } else {
    for (size_t i = at; i < bytes; ++i) dst[i - at] = 0;
  }
}

__global__ void cast_f32_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, size_t n) {
  chain_begin();
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    dst[i] = __float2bfloat16_rn(src[i]);
}

// ------------------------------------------------------------------ embedding
__global__ void embedding_fwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                                     __nv_bfloat16* __restrict__ out, int T, int D) {
  chain_begin();
  const int per_row = D / 8;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < static_cast<size_t>(T) * per_row;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t t = i / per_row, c = (i - t * per_row) * 8;
    *reinterpret_cast<bf16x8*>(out + t * D + c) =
        *reinterpret_cast<const bf16x8*>(table + static_cast<size_t>(ids[t]) * D + c);
  }
}
// grad[ids[t]] += dy[t], bound by the additions in L2.  VECTOR: four columns per addition, for gradients on a 16-byte
// boundary; one by one 16384 x 4096 took 376 us, this way 130; 4096 x
// 1024 24.5, 6.9.
template <bool VECTOR>
__global__ void embedding_bwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ dy,
                                     float* __restrict__ grad, int T, int D) {
  chain_begin();
  const int per_row = D / 8;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < static_cast<size_t>(T) * per_row;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t t = i / per_row, c = (i - t * per_row) * 8;
    float v[8];
    unpack8(*reinterpret_cast<const bf16x8*>(dy + t * D + c), v);
    float* dst = grad + static_cast<size_t>(ids[t]) * D + c;
    if (VECTOR) {
      atomicAdd(reinterpret_cast<float4*>(dst), make_float4(v[0], v[1], v[2], v[3]));
      atomicAdd(reinterpret_cast<float4*>(dst) + 1, make_float4(v[4], v[5], v[6], v[7]));
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) atomicAdd(dst + j, v[j]);
    }
  }
}

// ------------------------------------------------------------------ RoPE (adjacent pairs), in place
// x: [B, S, H, hd] with token pitch ``pitch`` elements (a view into the fused QKV buffer); rotates heads
// [0, H).  sign = +1 forward, -1 backward (the transpose rotation).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, int tokens, int S, int H, int hd, long long pitch,
                            float sign) {
  chain_begin();
  const int vec_per_head = hd / 8;
  const size_t total = static_cast<size_t>(tokens) * H * vec_per_head;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int v = static_cast<int>(i % vec_per_head);
    const int h = static_cast<int>((i / vec_per_head) % H);
    const size_t tok = i / (static_cast<size_t>(vec_per_head) * H);
    const int pos = static_cast<int>(tok % S);
    __nv_bfloat16* ptr = x + tok * pitch + static_cast<size_t>(h) * hd + v * 8;
    float f[8];
    unpack8(*reinterpret_cast<const bf16x8*>(ptr), f);
    const float4 c = *reinterpret_cast<const float4*>(cos_t + static_cast<size_t>(pos) * (hd / 2) + v * 4);
    float4 s = *reinterpret_cast<const float4*>(sin_t + static_cast<size_t>(pos) * (hd / 2) + v * 4);
    s.x *= sign; s.y *= sign; s.z *= sign; s.w *= sign;
    const float cc[4] = {c.x, c.y, c.z, c.w}, sn[4] = {s.x, s.y, s.z, s.w};
    float o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[2 * j] = f[2 * j] * cc[j] - f[2 * j + 1] * sn[j];
      o[2 * j + 1] = f[2 * j] * sn[j] + f[2 * j + 1] * cc[j];
    }
    *reinterpret_cast<bf16x8*>(ptr) = pack8(o);
  }
}

// The rotation of q [tokens, Hq*128] and k [tokens, Hkv*128] (token pitches ``q_pitch``, ``k_pitch``) into contiguous
// copies, one launch and one pass over each: bound by memory traffic (32 us at 8192 tokens of 32 + 8 heads; clones
// followed by rotations in place moved every element twice, 70 us in four launches).
__global__ void __launch_bounds__(256) rope_copy_kernel(const __nv_bfloat16* __restrict__ q,
                                                        const __nv_bfloat16* __restrict__ k,
                                                        __nv_bfloat16* __restrict__ q_out,
                                                        __nv_bfloat16* __restrict__ k_out,
                                                        const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                                        int tokens, int S, int Hq, int Hkv, long long q_pitch,
                                                        long long k_pitch) {
  chain_begin();
  const int per_token = (Hq + Hkv) * 16;       // 16-byte vectors
  const size_t total = static_cast<size_t>(tokens) * per_token;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t tok = i / per_token;
    int c = static_cast<int>(i - tok * per_token);
    const int pos = static_cast<int>(tok % S);
    const bool second = c >= Hq * 16;
    if (second) c -= Hq * 16;
    const __nv_bfloat16* src = second ? k + tok * k_pitch : q + tok * q_pitch;
    __nv_bfloat16* dst = second ? k_out + tok * Hkv * 128 : q_out + tok * Hq * 128;
    float f[8], o[8];
    unpack8(*reinterpret_cast<const bf16x8*>(src + c * 8), f);
    const float4 cc = *reinterpret_cast<const float4*>(cos_t + static_cast<size_t>(pos) * 64 + (c & 15) * 4);
    const float4 ss = *reinterpret_cast<const float4*>(sin_t + static_cast<size_t>(pos) * 64 + (c & 15) * 4);
    const float cv[4] = {cc.x, cc.y, cc.z, cc.w}, sv[4] = {ss.x, ss.y, ss.z, ss.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[2 * j] = f[2 * j] * cv[j] - f[2 * j + 1] * sv[j];
      o[2 * j + 1] = f[2 * j] * sv[j] + f[2 * j + 1] * cv[j];
    }
    *reinterpret_cast<bf16x8*>(dst + c * 8) = pack8(o);
  }
}

// SM count of the current device (grids are sized as a multiple of it).
static inline int sm_count_ew() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return sms;
}
static inline int grid_for(size_t work, int threads, int per_sm = 16) {
  size_t blocks = (work + threads - 1) / threads;
  if (blocks < 1) blocks = 1;
  const size_t cap = static_cast<size_t>(sm_count_ew()) * per_sm;
  return static_cast<int>(blocks > cap ? cap : blocks);
}
static inline int ok() { return cudaGetLastError() == cudaSuccess ? 0 : -1; }

constexpr int NORM_FWD_CTAS = 3;
constexpr int NORM_SMEM = 110 * 1024;        // two CTAs per SM
template <int N> struct Int { static constexpr int value = N; };
static inline int norm_rows_at_once(int D) { return D <= 512 ? 8 : D <= 1024 ? 4 : D <= 2048 ? 2 : 1; }
// ``launch(W, V, shared memory, ring stages)`` for rows of D columns and ``tensors`` tensors in the ring.
template <typename F>
static int launch_norm(int D, int tensors, F launch) {
  const int slot = norm_rows_at_once(D) * D * 2 * tensors;
  const int stages = min(NORM_RING, NORM_SMEM / slot);
  // (backward: the sums of the rows at once, four bytes a column, fit into one stage of three tensors)
  const int smem = max(stages, 1) * slot;
  if (D <= 512) return launch(Int<1>{}, Int<NORM_VECS>{}, smem, stages);
  if (D <= 1024) return launch(Int<2>{}, Int<NORM_VECS>{}, smem, stages);
  if (D <= 2048) return launch(Int<4>{}, Int<NORM_VECS>{}, smem, stages);
  if (D <= 4096) return launch(Int<8>{}, Int<NORM_VECS>{}, smem, stages);
  return launch(Int<8>{}, Int<4>{}, smem, stages);
}
template <int W, int V, int KIND, typename K>
static int norm_smem(K kernel) {
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NORM_SMEM) != cudaSuccess) return -3;
    set = true;
  }
  return 0;
}

}  // namespace b2

using namespace b2;
typedef __nv_bfloat16 bf16;

extern "C" {

// bf16 tensors: 16-byte aligned, rows of D elements one after the other.  status: device word, set if a copy did not arrive.
int b2_rmsnorm_fwd(const void* x, const void* delta, const float* w, void* sum_out, void* y, float* rstd, int rows,
                   int D, float eps, int* status, cudaStream_t s) {
  if (D % 8 || D > NORM_MAX_D) return -10;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(delta)) % 16) return -12;
  const int at_once = norm_rows_at_once(D);
  if ((rows + at_once - 1) / at_once <= sm_count_ew() * NORM_FWD_CTAS) {
    auto kernel = D <= 2048 ? rmsnorm_fwd_row_kernel<1> : D <= 4096 ? rmsnorm_fwd_row_kernel<2> : rmsnorm_fwd_row_kernel<4>;
    launch_next(kernel, min(rows, sm_count_ew() * 8), NORM_THREADS, 0, s, (const bf16*)x, (const bf16*)delta, w, (bf16*)sum_out,
                (bf16*)y, rstd, rows, D, eps);
    return ok();
  }
  return launch_norm(D, 2, [&](auto W, auto V, int smem, int stages) {
    auto kernel = rmsnorm_fwd_kernel<decltype(W)::value, decltype(V)::value>;
    if (const int rc = norm_smem<decltype(W)::value, decltype(V)::value, 0>(kernel)) return rc;
    launch_next(kernel, sm_count_ew() * NORM_FWD_CTAS, NORM_THREADS + 32, smem, s, (const bf16*)x, (const bf16*)delta, w,
                (bf16*)sum_out, (bf16*)y, rstd, status, rows, D, eps, stages);
    return ok();
  });
}

// dw_partial: fp32 [parts, D] scratch with parts = b2_rmsnorm_bwd_parts(rows, D); dw: fp32 [D] (overwritten).  dx may be residual:
// one CTA holds a row of all tensors before it stores that row.
// One wave, and as few partial rows as possible for the column sum: two CTAs are resident per SM, beyond 4096 columns one
// (registers; with twice as many 1024 x 8192 took 24.3 us instead of 19.7, 16384 x 8192 218 instead of 209).
int b2_rmsnorm_bwd_parts(int rows, int D) {
  const int R = norm_rows_at_once(D);
  return min((rows + R - 1) / R, sm_count_ew() * (D <= 4096 ? 2 : 1));
}
int b2_rmsnorm_bwd(const void* dy, const void* x, const float* w, const float* rstd, const void* residual, void* dx,
                   float* dw_partial, float* dw, int rows, int D, int* status, cudaStream_t s) {
  if (D % 8 || D > NORM_MAX_D) return -10;
  if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(residual)) % 16) return -12;
  const int parts = b2_rmsnorm_bwd_parts(rows, D), at_once = norm_rows_at_once(D);
  const int rc = launch_norm(D, 3, [&](auto W, auto V, int smem, int stages) {
    constexpr int w_ = decltype(W)::value, v_ = decltype(V)::value;
    if ((rows + at_once - 1) / at_once <= parts) {
      launch_next(rmsnorm_bwd_kernel<w_, v_, 0>, parts, NORM_THREADS, at_once * D * 4, s, (const bf16*)dy, (const bf16*)x, w, rstd,
                  (const bf16*)residual, (bf16*)dx, dw_partial, status, rows, D, stages);
      return ok();
    }
    auto kernel = rmsnorm_bwd_kernel<w_, v_, 1>;
    if (const int rc = norm_smem<w_, v_, 1>(kernel)) return rc;
    launch_next(kernel, parts, NORM_THREADS + 32, smem, s, (const bf16*)dy, (const bf16*)x, w, rstd, (const bf16*)residual,
                (bf16*)dx, dw_partial, status, rows, D, stages);
    return ok();
  });
  if (rc) return rc;
  if (parts <= 8) launch_next(column_sum_kernel<8>, (D + 31) / 32, 256, 0, s, dw_partial, dw, parts, D);
  else launch_next(column_sum_kernel<32>, (D + 31) / 32, 1024, 0, s, dw_partial, dw, parts, D);
  return ok();
}

}  // extern "C"

// One CTA covers 32 tokens per turn; at most two per SM, so that the weights are staged once for many tokens.
static int skinny_grid(int T) { return min((T + 31) / 32, sm_count_ew() * 2); }

template <bool TOP2>
static int launch_skinny_nt(const void* x, const void* w, float* out, float* weights, long long* idx, float* probs, int T,
                            int N, int K, cudaStream_t s) {
  const size_t smem = static_cast<size_t>(N) * K * 2;
  if (smem > 200 * 1024) return -11;
  static bool set = false;
  if (!set) {
    cudaFuncSetAttribute(skinny_nt_kernel<8, TOP2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(skinny_nt_kernel<16, TOP2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    set = true;
  }
  auto kernel = N <= 8 ? skinny_nt_kernel<8, TOP2> : skinny_nt_kernel<16, TOP2>;
  launch_next(kernel, skinny_grid(T), 256, smem, s, (const bf16*)x, (const bf16*)w, out, weights, idx, probs, T, N, K);
  return ok();
}
extern "C" {
int b2_skinny_nt(const void* x, const void* w, float* out, int T, int N, int K, cudaStream_t s) {
  if (N > SKINNY_MAX_N || K % 8 || (N * K) % 8) return -10;
  return launch_skinny_nt<false>(x, w, out, nullptr, nullptr, nullptr, T, N, K, s);
}
// Router in one launch: the softmax ``probs`` [T,N] of x w^T, the two largest (idx) and their weights.
int b2_router_fwd(const void* x, const void* w, float* weights, long long* idx, float* probs, int T, int N, int K,
                  cudaStream_t s) {
  if (N < 2 || N > SKINNY_MAX_N || K % 8 || (N * K) % 8) return -10;
  return launch_skinny_nt<true>(x, w, nullptr, weights, idx, probs, T, N, K, s);
}
int b2_skinny_nn(const float* dy, const void* w, void* dx, int T, int N, int K, cudaStream_t s) {
  if (N > SKINNY_MAX_N || K % 8) return -10;
  const size_t smem = static_cast<size_t>(N) * K * 2;
  if (smem > 200 * 1024) return -11;
  static bool set = false;
  if (!set) {
    cudaFuncSetAttribute(skinny_nn_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(skinny_nn_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    set = true;
  }
  if (N <= 8) launch_next(skinny_nn_kernel<8>, skinny_grid(T), 256, smem, s, dy, (const bf16*)w, (bf16*)dx, T, N, K);
  else launch_next(skinny_nn_kernel<16>, skinny_grid(T), 256, smem, s, dy, (const bf16*)w, (bf16*)dx, T, N, K);
  return ok();
}
int b2_skinny_tn(const float* dy, const void* x, float* dw, int T, int N, int K, cudaStream_t s) {
  if (N > SKINNY_MAX_N || K % 8) return -10;
  if (T < 1) return 0;
  // two CTAs per SM (registers) over (columns, tokens), at least 64 tokens each
  const int columns = (K + 255) / 256;
  const int splits = max(1, min((T + 63) / 64, sm_count_ew() * 2 / columns));
  const int per = (T + splits - 1) / splits;
  const dim3 grid(columns, (T + per - 1) / per);
  if (N <= 8) launch_next(skinny_tn_kernel<8>, grid, 256, 0, s, dy, (const bf16*)x, dw, T, N, K, per);
  else launch_next(skinny_tn_kernel<16>, grid, 256, 0, s, dy, (const bf16*)x, dw, T, N, K, per);
  return ok();
}

int b2_router_top2_fwd(const float* logits, float* weights, long long* idx, float* probs, int T, int E,
                       cudaStream_t s) {
  if (E > ROUTER_MAX_E || E < 2) return -10;
  launch_next(router_top2_fwd_kernel, (T + 127) / 128, 128, 0, s, logits, weights, idx, probs, T, E);
  return ok();
}
int b2_router_top2_bwd(const float* dweights, const float* probs, const long long* idx, const float* weights,
                       float* dlogits, int T, int E, cudaStream_t s) {
  launch_next(router_top2_bwd_kernel, (T + 127) / 128, 128, 0, s, dweights, probs, idx, weights, dlogits, T, E);
  return ok();
}

int b2_swiglu_bwd(const void* dh, const void* gate, const void* up, void* dgu, void* h, const int* live_rows, int rows,
                  int F, cudaStream_t s) {
  if (F % 8) return -10;
  launch_next(swiglu_bwd_kernel, grid_for(static_cast<size_t>(rows) * F / 8, 256), 256, 0, s, (const bf16*)dh, (const bf16*)gate,
              (const bf16*)up, (bf16*)dgu, (bf16*)h, live_rows, rows, F);
  return ok();
}

// ``loss`` (zeroed by the caller; fp32, or a double where ``wide``) += loss_scale * sum of the rows' losses, logits <-
// grad_scale * gradient; rows up to 32768 entries are read once and written once.
int b2_cross_entropy2(void* logits, const long long* targets, void* loss, int wide, int T, int V, float loss_scale,
                      float grad_scale, int* status, cudaStream_t s) {
  if (V % 8) return -10;
  if (V > CE_THREADS * 8 * CE_REG_CHUNKS && loss_scale != grad_scale) return -11;   // the streaming kernel has one scale
  if (V <= CE_THREADS * 8 * CE_REG_CHUNKS) {
    // one wave of resident CTAs, so that every CTA has a next row to request while it works on one
    const int grid = min(T, sm_count_ew() * 2);
    if (V <= CE_THREADS * 32) {
      auto kernel = V <= CE_THREADS * 16 ? cross_entropy_reg_kernel<2> : cross_entropy_reg_kernel<4>;
      launch_next(kernel, grid, CE_THREADS, 0, s, (bf16*)logits, targets, loss, wide, T, V, loss_scale, grad_scale);
      return ok();
    }
    static bool set = false;
    if (!set) {
      if (cudaFuncSetAttribute(cross_entropy_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536) != cudaSuccess)
        return -3;
      set = true;
    }
    launch_next(cross_entropy_bulk_kernel, grid, CE_THREADS, V * 2, s, (bf16*)logits, targets, loss, wide, status, T, V, loss_scale,
                                                              grad_scale);
    return ok();
  }
  launch_next(cross_entropy_kernel, min(T, sm_count_ew() * 4), CE_THREADS, 0, s, (bf16*)logits, targets, loss, wide, T, V,
              loss_scale);
  return ok();
}
int b2_scale_bf16(void* x, const float* factor, long long n, cudaStream_t s) {
  if (n % 8) return -10;
  launch_next(scale_bf16_kernel, grid_for(n / 8, 256), 256, 0, s, (bf16*)x, factor, n / 8);
  return ok();
}

// ``count`` tensors of the same types: ``ptrs`` holds p, g, m, v and the optional bf16 copy (0 for none) of each, ``n``
// the element counts.  dtype codes: 0 fp32, 1 bf16.
int b2_adamw(const unsigned long long* ptrs, const long long* n, int count, int p_dt, int g_dt, int s_dt, float lr,
             float beta1, float beta2, float eps, float wd, float a_t, float grad_scale, cudaStream_t s) {
  const int code = p_dt * 4 + g_dt * 2 + s_dt;
  if (code < 0 || code > 7) return -10;
  for (int base = 0; base < count; base += ADAMW_MAX) {
    AdamwTable table;
    table.count = min(ADAMW_MAX, count - base);
    long long chunks = 0, total = 0;
    for (int i = 0; i < table.count; ++i) total += n[base + i];
    table.chunk = total < static_cast<long long>(sm_count_ew()) * 16 * ADAMW_CHUNK ? ADAMW_SMALL_CHUNK : ADAMW_CHUNK;
    for (int i = 0; i < table.count; ++i) {
      const unsigned long long* q = ptrs + 5 * (base + i);
      table.t[i] = {reinterpret_cast<void*>(q[0]), reinterpret_cast<const void*>(q[1]), reinterpret_cast<void*>(q[2]),
                    reinterpret_cast<void*>(q[3]), reinterpret_cast<bf16*>(q[4]), n[base + i]};
      table.first_chunk[i] = static_cast<int>(chunks);
      chunks += (n[base + i] + table.chunk - 1) / table.chunk;
      if (chunks > 0x7fffffffLL) return -11;
    }
    table.first_chunk[table.count] = static_cast<int>(chunks);
    if (chunks == 0) continue;
    const int grid = static_cast<int>(min(chunks, static_cast<long long>(sm_count_ew()) * 16));
#define B2_ADAMW(P, G, S) launch_next(adamw_kernel<P, G, S>, grid, 256, 0, s, table, lr, beta1, beta2, eps, wd, a_t, grad_scale)
    switch (code) {
      case 0: B2_ADAMW(float, float, float); break;
      case 1: B2_ADAMW(float, float, bf16); break;
      case 2: B2_ADAMW(float, bf16, float); break;
      case 3: B2_ADAMW(float, bf16, bf16); break;
      case 4: B2_ADAMW(bf16, float, float); break;
      case 5: B2_ADAMW(bf16, float, bf16); break;
      case 6: B2_ADAMW(bf16, bf16, float); break;
      default: B2_ADAMW(bf16, bf16, bf16); break;
    }
#undef B2_ADAMW
    if (ok()) return -1;
  }
  return 0;
}
// ``ptrs``: 16-byte aligned buffers of ``bytes`` bytes each.
int b2_zero(const unsigned long long* ptrs, const long long* bytes, int count, cudaStream_t s) {
  for (int base = 0; base < count; base += ZERO_MAX) {
    ZeroTable table;
    table.count = min(ZERO_MAX, count - base);
    long long chunks = 0;
    for (int i = 0; i < table.count; ++i) {
      if (ptrs[base + i] % 16) return -10;
      table.p[i] = reinterpret_cast<uint8_t*>(ptrs[base + i]);
      table.bytes[i] = bytes[base + i];
      table.first_chunk[i] = static_cast<int>(chunks);
      chunks += (bytes[base + i] + ZERO_CHUNK - 1) / ZERO_CHUNK;
      if (chunks > 0x7fffffffLL) return -11;
    }
    table.first_chunk[table.count] = static_cast<int>(chunks);
    if (chunks == 0) continue;
    launch_next(zero_kernel, static_cast<unsigned>(chunks), 256, 0, s, table);
    if (ok()) return -1;
  }
  return 0;
}
int b2_cast_f32_bf16(const float* src, void* dst, long long n, cudaStream_t s) {
  launch_next(cast_f32_bf16_kernel, grid_for(n, 256, 32), 256, 0, s, src, (bf16*)dst, n);
  return ok();
}

int b2_embedding_fwd(const long long* ids, const void* table, void* out, int T, int D, cudaStream_t s) {
  if (D % 8) return -10;
  launch_next(embedding_fwd_kernel, grid_for(static_cast<size_t>(T) * D / 8, 256), 256, 0, s, ids, (const bf16*)table,
                                                                                    (bf16*)out, T, D);
  return ok();
}
int b2_embedding_bwd(const long long* ids, const void* dy, float* grad, int T, int D, cudaStream_t s) {
  if (D % 8) return -10;
  auto kernel = reinterpret_cast<uintptr_t>(grad) % 16 == 0 ? embedding_bwd_kernel<true> : embedding_bwd_kernel<false>;
  launch_next(kernel, grid_for(static_cast<size_t>(T) * D / 8, 256), 256, 0, s, ids, (const bf16*)dy, grad, T, D);
  return ok();
}

int b2_rope(void* x, const float* cos_t, const float* sin_t, int tokens, int S, int H, int hd, long long pitch,
            float sign, cudaStream_t s) {
  if (hd % 8 || pitch % 8) return -10;
  launch_next(rope_kernel, grid_for(static_cast<size_t>(tokens) * H * hd / 8, 256), 256, 0, s, (bf16*)x, cos_t, sin_t, tokens, S,
                                                                                     H, hd, pitch, sign);
  return ok();
}

int b2_rope_copy(const void* q, const void* k, void* q_out, void* k_out, const float* cos_t, const float* sin_t,
                 int tokens, int S, int Hq, int Hkv, long long q_pitch, long long k_pitch, cudaStream_t s) {
  if (q_pitch % 8 || k_pitch % 8 || S < 1) return -10;
  launch_next(rope_copy_kernel, grid_for(static_cast<size_t>(tokens) * (Hq + Hkv) * 16, 256), 256, 0, s, (const bf16*)q,
              (const bf16*)k, (bf16*)q_out, (bf16*)k_out, cos_t, sin_t, tokens, S, Hq, Hkv, q_pitch, k_pitch);
  return ok();
}

}  // extern "C"

namespace b2 {
// The device-wide nanosecond clock, stored when the stream reaches this launch: two of these bracket a region
// with one clock for every SM (CUDA events measure the same span; this form can be read by other kernels too).
__global__ void timestamp_kernel(unsigned long long* out) {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  *out = t;
}
}  // namespace b2

extern "C" int b2_device_timestamp(unsigned long long* out, cudaStream_t s) {
  b2::timestamp_kernel<<<1, 1, 0, s>>>(out);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
