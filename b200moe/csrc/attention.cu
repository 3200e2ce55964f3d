// Causal grouped-query flash attention for head_dim 128 on tcgen05 tensor cores:
// forward, and the backward pass as two kernels (dK/dV per key tile, dQ per query
// tile).  Inputs are bf16 views [B, S, H, 128] with a common token pitch (the fused
// QKV projection, already rotated by the RoPE kernel); Q/K/V/dO tiles come in by TMA
// (plain per-CTA tile loads) in the 128-byte-swizzled layout, so the same
// shared-memory tile serves as a K-major or an MN-major MMA operand.  Scores and
// probabilities live in tensor memory: S = Q K^T lands in TMEM, the softmax warps turn
// it into bf16 P in place, and P feeds the next MMA straight from TMEM (A operand in
// tensor memory), so P never touches shared memory.
//
// Forward, one CTA per (256 queries, head, batch), or per 128 queries in grids of one wave: see attn_fwd_kernel and
//   attn_fwd_one_tile_kernel.
// Backward dK/dV, one CTA per (128 keys, kv head, batch): loops over the 4 query heads
//   of the group and their causal query tiles with S^T = K Q^T, dP^T = V dO^T, so P^T
//   and dS^T are A operands in TMEM; dV and dK accumulate in TMEM over the whole loop
//   (the GQA reduction needs no atomics).
// Backward dQ, one CTA per (128 queries, head, batch): recomputes S and dP per key tile
//   and accumulates dQ += dS K in TMEM.
// A sequence may have any length: its last tile reads zeros behind it and is masked.
// Every barrier wait is bounded; a wait that runs out sets the status word.
#include "chain.cuh"
#include "entries.h"
#include "ptx.cuh"
#include "tensormap.cuh"

#include <atomic>

namespace b2 {

constexpr int HD = 128;
constexpr int TQ = 128;
constexpr int TK = 128;
constexpr int TILE_BYTES = 128 * HD * 2;      // 32 KiB: two swizzle atoms of [128 rows x 64 cols]
constexpr int ATOM_BYTES = 16384;
constexpr int ATTN_THREADS = 320;       // two softmax warpgroups, TMA warp, MMA warp

struct AttnParams {
  CUtensorMap map_q, map_k, map_v, map_do;
  int B, S, Hq, Hkv;
  int causal;             // 1: keys after the query are masked; 0: every query sees every key
  float scale;            // 1/sqrt(head_dim)
  float scale_log2;       // scale * log2(e)
  int set_heads;          // heads that share a launch-order set (attn_work)
  void* out;              // forward: [B,S,Hq,128] contiguous, in the type of q, k, v
  float* lse;             // [B,Hq,S] natural-log row sums (forward writes)
  const float* stats;     // backward: [B*Hq][2][Sp] with Sp = S rounded up to 128: -lse * log2(e), then -rowsum(dO * O);
                          // -inf and 0 behind the sequence (such queries get zero probabilities)
  __nv_bfloat16* dq;      // [B,S,Hq,128]
  __nv_bfloat16* dk;      // [B,S,Hkv,128]
  __nv_bfloat16* dv;      // [B,S,Hkv,128]
  long long dq_pitch, dk_pitch, dv_pitch;   // elements per token of the gradient outputs
  const float* rope_cos;  // backward, optional: [S, 64] tables of the rotation that was applied to q and k before the
  const float* rope_sin;  // forward pass; dq and dk are then stored rotated back (gradients of the unrotated q, k)
  int* status;
};

// Transposed rotary embedding on 32 consecutive columns (16 adjacent pairs) of one head, in registers:
// (d0, d1) -> (d0 c + d1 s, d1 c - d0 s).  ``first_pair`` = (column of a[0] within the head) / 2.
__device__ __forceinline__ void unrotate32(uint32_t (&a)[32], const float* cos_t, const float* sin_t, size_t pos,
                                           int first_pair) {
  const float4* c4 = reinterpret_cast<const float4*>(cos_t + pos * 64 + first_pair);
  const float4* s4 = reinterpret_cast<const float4*>(sin_t + pos * 64 + first_pair);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 cc = c4[q], ss = s4[q];
    const float cv[4] = {cc.x, cc.y, cc.z, cc.w}, sv[4] = {ss.x, ss.y, ss.z, ss.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float d0 = __uint_as_float(a[8 * q + 2 * j]), d1 = __uint_as_float(a[8 * q + 2 * j + 1]);
      a[8 * q + 2 * j] = __float_as_uint(d0 * cv[j] + d1 * sv[j]);
      a[8 * q + 2 * j + 1] = __float_as_uint(d1 * cv[j] - d0 * sv[j]);
    }
  }
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// K-major operand inside a [128 x 128] tile stored as two atoms: 16-element k-step ks (0..7).
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile, int ks) {
  return umma_smem_desc(tile + (ks >> 2) * ATOM_BYTES + (ks & 3) * 32, 16, 1024);
}
// The same tile read as an MN-major operand: MN runs along the 128 columns (two 64-column atoms,
// ATOM_BYTES apart), K along the rows; k-step ks covers rows [16 ks, 16 ks + 16).
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t tile, int ks) {
  return umma_smem_desc(tile + ks * 2048, ATOM_BYTES, 1024);
}

// 128 tokens x 128 columns of one batch entry; tokens behind the sequence read as zeros.
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col0, int token0,
                                          int batch) {
  tma_load_3d(dst, map, bar, col0, token0, batch);
  tma_load_3d(dst + ATOM_BYTES, map, bar, col0 + 64, token0, batch);
}

template <int F16>
constexpr uint32_t attn_idesc(int b_mn_major) {
  return F16 ? umma_idesc_f16(128, 128, 0, b_mn_major) : umma_idesc_bf16(128, 128, 0, b_mn_major);
}

// Two fp32 values in a 64-bit register: one instruction of the FMA pipe works on both (same rounding as two).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 make_f32x2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f32x2 bits_f32x2(const uint32_t* two) {
  return make_f32x2(__uint_as_float(two[0]), __uint_as_float(two[1]));
}
__device__ __forceinline__ void split_f32x2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma_f32x2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add_f32x2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul_f32x2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ float sum_f32x2(f32x2 v) {
  float a, b;
  split_f32x2(v, a, b);
  return a + b;
}

// Of ``count`` copies that a producer has issued into a ring of SLOTS barriers, the last on each slot: a CTA that gives up
// waits for them (with a limit) before its shared memory goes to another one.
template <int SLOTS>
__device__ __forceinline__ void drain_ring(uint64_t* full, int count) {
  for (int i = count > SLOTS ? count - SLOTS : 0; i < count; ++i) mbar_wait(&full[i % SLOTS], (i / SLOTS) & 1);
}

#define ATTN_FAIL(code)            \
  {                                \
    *abort_flag = 1;               \
    atomicExch(p.status, code);    \
  }

// ================================================================= forward
struct FwdBars {
  uint64_t q_full, k_full[2], v_full[2], k_empty[2], v_empty[2], s_full[2], p_lo[2], p_hi[2], o_done[2];
};

// The two-tile kernel's threads: two softmax warpgroups and one with the TMA and the MMA warp.  At launch each thread has 168
// registers; the softmax threads, which hold 128 scores, take most of the third warpgroup's.
constexpr int FWD_THREADS = 384, FWD_SOFTMAX_REGS = 208, FWD_PRODUCER_REGS = 88;
static_assert(256 * FWD_SOFTMAX_REGS + 128 * FWD_PRODUCER_REGS <= 384 * 168, "registers of the forward CTA");
template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// Which tile a CTA works on.  CTAs are numbered so that the longest causal rows of a set of heads start first, and a
// set holds as many heads as keep the tensors they re-read inside the L2 (p.set_heads, host side).
struct AttnWork {
  int tile, head;          // 0 = longest; flattened batch * heads + head
};
__device__ __forceinline__ AttnWork attn_work(const AttnParams& p, int tiles, int heads, int index) {
  const int per_set = p.set_heads * tiles;
  const int set = index / per_set;
  const int rest = index - set * per_set;
  const int count = min(p.set_heads, heads - set * p.set_heads);
  return {rest / count, set * p.set_heads + rest % count};
}

// Probabilities of 64 scores of one row: exponentials, stored in 16 bits as pairs over the first 32 of the 64 score
// columns at ``ts`` (which the thread has read before), and their sum.  Both forward kernels call it, so the order of the
// sum (eight partial sums: no long add chain) is the same in both, and which of them runs does not change a bit of the
// result (for the two-tile kernel a second sum per row and tile, 82.0 -> 82.3 us at 32 heads of 2048 tokens, every key).
// CHUNK columns are stored at a time: 64 leave no bubble before a store, 32 need fewer registers.
template <int F16, int CHUNK>
__device__ __forceinline__ float probabilities64(const uint32_t (&lo)[32], const uint32_t (&hi)[32], uint32_t ts,
                                                 float scale_log2, float neg) {
  const f32x2 scale2 = make_f32x2(scale_log2, scale_log2), neg2 = make_f32x2(neg, neg);
  f32x2 sum2[4] = {0, 0, 0, 0};
  uint32_t packed[CHUNK / 2];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    float x0, x1;
    split_f32x2(fma_f32x2(bits_f32x2(&(i < 16 ? lo : hi)[(i & 15) * 2]), scale2, neg2), x0, x1);
    const float p0 = ex2(x0), p1 = ex2(x1);
    sum2[i & 3] = add_f32x2(sum2[i & 3], make_f32x2(p0, p1));
    packed[i % (CHUNK / 2)] = F16 ? pack_f16(p0, p1) : pack_bf16(p0, p1);
    if constexpr (CHUNK == 32) {
      if (i % 16 == 15) tmem_st_32x16(ts + i / 16 * 16, packed);
    }
  }
  if constexpr (CHUNK == 64) tmem_st_32x32(ts, packed);
  return sum_f32x2(add_f32x2(add_f32x2(sum2[0], sum2[1]), add_f32x2(sum2[2], sum2[3])));
}

// Stores 32 output columns of one row, normalised.
template <int F16>
__device__ __forceinline__ void store_out32(uint8_t* dst, const uint32_t (&o)[32], float inv) {
  uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float a = __uint_as_float(o[8 * i + 2 * k]) * inv, e = __uint_as_float(o[8 * i + 2 * k + 1]) * inv;
      w[k] = F16 ? pack_f16(a, e) : pack_bf16(a, e);
    }
    d4[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// One CTA per (two adjacent 128-query tiles, head, batch): the tiles ping-pong, so the tensor core works on one while
// the softmax warpgroup of the other turns scores into probabilities.  A thread owns a whole query row (128 score
// columns in registers): no exchange of row maxima, one barrier per half of a probability tile.  S and O of both tiles
// fill tensor memory; P overwrites S.  MMA order O0(j) S0(j+1) O1(j) S1(j+1): a tile's next scores are issued behind
// the product that still reads its probabilities, so "scores ready" also means "output of the previous key tile
// accumulated", and the rare rescale of O (row maximum grew by more than 2^8) needs no further wait.
// Bound by the chain scores -> exponentials -> product of each tile: of 2930 cycles per key tile 360 were the row maximum, now
// formed beside the first half's exponentials, and 2048 are the products of both tiles.  32/8 heads of 8192 tokens, causal:
// 447 -> 434 us, 1270 TFLOP/s (one query tile per CTA with two threads per row: 622 us); 32 heads of 2048 tokens, every key,
// fp16: 70.7 -> 68.6 us (at 1.9 GHz; 78 -> 76 on a slower box).  The special-function unit is not the limit: an eighth to
// half of the exponentials as polynomials on the FMA pipe took 1 to 18 % longer; nor do scores in two halves of 64 keys help,
// whose products read their operands from shared memory half as often as they use them (2930 -> 3350 cycles).
template <int F16>
__global__ void __launch_bounds__(FWD_THREADS, 1) attn_fwd_kernel(const __grid_constant__ AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  uint8_t* sQ = smem;                       // 2 tiles
  uint8_t* sK = sQ + 2 * TILE_BYTES;        // 2 stages
  uint8_t* sV = sK + 2 * TILE_BYTES;        // 2 stages
  FwdBars* bars = reinterpret_cast<FwdBars*>(sV + 2 * TILE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv_tiles = (p.S + TK - 1) / TK;
  const int pairs = (kv_tiles + 1) / 2;
  const AttnWork work = attn_work(p, pairs, p.B * p.Hq, static_cast<int>(blockIdx.x));
  const int qt0 = 2 * (pairs - 1 - work.tile);
  const int b = work.head / p.Hq, h = work.head - b * p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  // key tiles that each of the two query tiles sees (the second one may lie behind the sequence)
  const int n0 = p.causal ? qt0 + 1 : kv_tiles;
  const int n1 = qt0 + 1 >= kv_tiles ? 0 : (p.causal ? qt0 + 2 : kv_tiles);
  const int n_kv = max(n0, n1);

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->k_full[s], 1);
      mbar_init(&bars->v_full[s], 1);
      mbar_init(&bars->k_empty[s], 1);
      mbar_init(&bars->v_empty[s], 1);
      mbar_init(&bars->s_full[s], 1);
      mbar_init(&bars->p_lo[s], 4);
      mbar_init(&bars->p_hi[s], 4);
      mbar_init(&bars->o_done[s], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_begin();
  const uint32_t tmem = *tmem_slot;         // S0 | S1 | O0 | O1, 128 columns each

  if (warp >= 8) {
    reg_dec<FWD_PRODUCER_REGS>();
    if (warp == 8 && elect_one()) {
      mbar_expect_tx(&bars->q_full, (n1 ? 2 : 1) * TILE_BYTES);
      load_tile(sQ, &p.map_q, &bars->q_full, h * HD, qt0 * TQ, b);
      if (n1) load_tile(sQ + TILE_BYTES, &p.map_q, &bars->q_full, h * HD, (qt0 + 1) * TQ, b);
      int j = 0, key_ahead = 0;
      for (; j < n_kv && !*abort_flag; ++j) {
        const int s = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        if (!mbar_wait(&bars->k_empty[s], ph)) { ATTN_FAIL(201); break; }
        mbar_expect_tx(&bars->k_full[s], TILE_BYTES);
        load_tile(sK + s * TILE_BYTES, &p.map_k, &bars->k_full[s], hk * HD, j * TK, b);
        if (!mbar_wait(&bars->v_empty[s], ph)) { ATTN_FAIL(202); key_ahead = 1; break; }
        mbar_expect_tx(&bars->v_full[s], TILE_BYTES);
        load_tile(sV + s * TILE_BYTES, &p.map_v, &bars->v_full[s], hk * HD, j * TK, b);
      }
      if (*abort_flag) {
        mbar_wait(&bars->q_full, 0);
        drain_ring<2>(bars->k_full, j + key_ahead);
        drain_ring<2>(bars->v_full, j);
      }
    }
    if (warp == 9 && elect_one()) {
      constexpr uint32_t idesc_qk = attn_idesc<F16>(0);
      constexpr uint32_t idesc_pv = attn_idesc<F16>(1);
      auto issue_s = [&](int t, int j) {
        const uint32_t q_addr = smem_u32(sQ + t * TILE_BYTES), k_addr = smem_u32(sK + (j & 1) * TILE_BYTES);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16_ss(tmem + t * 128, desc_kmajor(q_addr, ks), desc_kmajor(k_addr, ks), idesc_qk, ks != 0);
        umma_commit(&bars->s_full[t]);
      };
      bool ok = mbar_wait(&bars->q_full, 0) && mbar_wait(&bars->k_full[0], 0);
      if (!ok) ATTN_FAIL(203);
      if (ok) {
        tc_fence_after();
        issue_s(0, 0);
        if (n1) issue_s(1, 0);
        umma_commit(&bars->k_empty[0]);
      }
      for (int j = 0; j < n_kv && ok && !*abort_flag; ++j) {
        const uint32_t ph = j & 1;
        if (!mbar_wait(&bars->v_full[j & 1], (j >> 1) & 1) ||
            (j + 1 < n_kv && !mbar_wait(&bars->k_full[(j + 1) & 1], ((j + 1) >> 1) & 1))) {
          ATTN_FAIL(204);
          break;
        }
        const uint32_t v_addr = smem_u32(sV + (j & 1) * TILE_BYTES);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int n = t ? n1 : n0;
          if (j >= n || !ok) continue;
          if (!mbar_wait(&bars->p_lo[t], ph)) { ok = false; continue; }
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16_ts(tmem + 256 + t * 128, tmem + t * 128 + ks * 8, desc_mnmajor(v_addr, ks), idesc_pv, (j | ks) != 0);
          if (!mbar_wait(&bars->p_hi[t], ph)) { ok = false; continue; }
          tc_fence_after();
#pragma unroll
          for (int ks = 4; ks < 8; ++ks)
            umma_bf16_ts(tmem + 256 + t * 128, tmem + t * 128 + ks * 8, desc_mnmajor(v_addr, ks), idesc_pv, 1);
          if (j + 1 == n) umma_commit(&bars->o_done[t]);
          else issue_s(t, j + 1);
        }
        if (!ok) { ATTN_FAIL(205); break; }
        umma_commit(&bars->v_empty[j & 1]);
        if (j + 1 < n_kv) umma_commit(&bars->k_empty[(j + 1) & 1]);
      }
    }
  } else {
    reg_inc<FWD_SOFTMAX_REGS>();
    const int t = warp >> 2;                              // query tile of this warpgroup
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                       // query row inside the tile
    const int qt = qt0 + t;
    const int n = t ? n1 : n0;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t ts = tmem + t * 128 + lane_base, to = tmem + 256 + t * 128 + lane_base;
    float m_ref = -INFINITY;
    float l[2] = {0.f, 0.f};                              // row sums of the two column halves
    for (int j = 0; j < n && !*abort_flag; ++j) {
      if (!mbar_wait(&bars->s_full[t], j & 1)) { ATTN_FAIL(206); break; }
      tc_fence_after();
      uint32_t raw[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(ts + c * 32, raw[c]);
      tmem_ld_wait();
      auto score = [&](int i) { return __uint_as_float(raw[i >> 5][i & 31]); };
      // keys that the row does not see: after the query (causal, diagonal tile) or behind the sequence
      const bool diagonal = p.causal && j == qt;
      if (diagonal || (j + 1) * TK > p.S) {
        const int limit = diagonal ? r + 1 : p.S - j * TK;
#pragma unroll
        for (int i = 0; i < 128; ++i)
          if (i >= limit) raw[i >> 5][i & 31] = 0xff800000u;   // -inf
      }
      auto row_max = [&] {
        float mpart[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 128; i += 2) mpart[(i >> 1) & 3] = fmaxf(fmaxf(mpart[(i >> 1) & 3], score(i)), score(i + 1));
        return fmaxf(fmaxf(fmaxf(mpart[0], mpart[1]), fmaxf(mpart[2], mpart[3])), m_ref);
      };
      if (j == 0) m_ref = row_max();
      // The first half's exponentials do not wait for the row maximum, which is formed beside them: the reference rarely
      // moves (by more than 2^8), and where it does they are formed again.
      float low = probabilities64<F16, 32>(raw[0], raw[1], ts, p.scale_log2, -m_ref * p.scale_log2);
      const float mx = row_max();
      if (__any_sync(0xffffffffu, (mx - m_ref) * p.scale_log2 > 8.f)) {
        const float alpha = ex2((m_ref - mx) * p.scale_log2);
        m_ref = mx;
        l[0] *= alpha;
        l[1] *= alpha;
#pragma unroll 1
        for (int c = 0; c < 8; ++c) {
          uint32_t o[16];
          tmem_ld_32x16(to + c * 16, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x16(to + c * 16, o);
        }
        low = probabilities64<F16, 32>(raw[0], raw[1], ts, p.scale_log2, -m_ref * p.scale_log2);
      }
      auto publish = [&](uint64_t* bar) {
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
      };
      l[0] += low;
      publish(&bars->p_lo[t]);
      l[1] += probabilities64<F16, 32>(raw[2], raw[3], ts + 32, p.scale_log2, -m_ref * p.scale_log2);
      publish(&bars->p_hi[t]);
    }
    // epilogue: normalise and store this thread's query row
    if (n > 0 && !*abort_flag) {
      if (!mbar_wait(&bars->o_done[t], 0)) ATTN_FAIL(208);
      tc_fence_after();
      const float sum = l[0] + l[1], inv = 1.f / sum;
      const int pos = qt * TQ + r;
      uint8_t* dst = static_cast<uint8_t*>(p.out) + ((static_cast<size_t>(b) * p.S + pos) * p.Hq + h) * HD * 2;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(to + c * 32, o);
        tmem_ld_wait();
        if (pos < p.S) store_out32<F16>(dst + c * 64, o, inv);
        __syncwarp();
      }
      if (pos < p.S) p.lse[static_cast<size_t>(work.head) * p.S + pos] = m_ref * p.scale + logf(sum);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// The same for grids of at most one CTA per SM: one CTA per (128 queries, head, batch), a row's 128 score columns shared by
// two threads (a warpgroup per 64 columns) that exchange their row maxima, scores of two key tiles in flight.  A tile's
// chain is half as long as with a row per thread, and where the two-tile form would leave half of the SMs idle that is
// all that counts: 32 heads of 512 tokens (128 CTAs) 9.9 us against 13.6, 4 heads of 4096 40.2 against 60.0; with 160
// CTAs, a second wave, 15.7 against 13.7.  Results are the same bit for bit.
struct FwdOneBars {
  uint64_t q_full, k_full[2], v_full[2], k_empty[2], v_empty[2], s_full[2], p_full[2], o_done, row_ready;
};
struct FwdOneSmem {
  uint8_t q[TILE_BYTES], k[2][TILE_BYTES], v[2][TILE_BYTES];
  float row_max[2][2][TQ], row_sum[2][TQ];      // [buffer][half][row], [half][row]
  FwdOneBars bars;
  uint32_t tmem_slot;
  int abort_flag;
};

template <int F16>
__global__ void __launch_bounds__(ATTN_THREADS, 1) attn_fwd_one_tile_kernel(const __grid_constant__ AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  FwdOneSmem& sm = *reinterpret_cast<FwdOneSmem*>(smem_raw);
  FwdOneBars* bars = &sm.bars;
  volatile int* abort_flag = &sm.abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv_tiles = (p.S + TK - 1) / TK;
  const AttnWork work = attn_work(p, kv_tiles, p.B * p.Hq, static_cast<int>(blockIdx.x));
  const int qt = kv_tiles - 1 - work.tile;
  const int b = work.head / p.Hq, h = work.head - b * p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  const int n_kv = p.causal ? qt + 1 : kv_tiles;

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->k_full[s], 1);
      mbar_init(&bars->v_full[s], 1);
      mbar_init(&bars->k_empty[s], 1);
      mbar_init(&bars->v_empty[s], 1);
      mbar_init(&bars->s_full[s], 1);
      mbar_init(&bars->p_full[s], 8);
    }
    mbar_init(&bars->o_done, 1);
    mbar_init(&bars->row_ready, 8);
    sm.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(&sm.tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_begin();
  const uint32_t tmem = sm.tmem_slot;       // S / P of even and odd key tiles, O: 128 columns each
  const uint32_t t_o = tmem + 256;

  if (warp == 8) {
    if (elect_one()) {
      mbar_expect_tx(&bars->q_full, TILE_BYTES);
      load_tile(sm.q, &p.map_q, &bars->q_full, h * HD, qt * TQ, b);
      int j = 0, key_ahead = 0;
      for (; j < n_kv && !*abort_flag; ++j) {
        const int s = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        if (!mbar_wait(&bars->k_empty[s], ph)) { ATTN_FAIL(201); break; }
        mbar_expect_tx(&bars->k_full[s], TILE_BYTES);
        load_tile(sm.k[s], &p.map_k, &bars->k_full[s], hk * HD, j * TK, b);
        if (!mbar_wait(&bars->v_empty[s], ph)) { ATTN_FAIL(202); key_ahead = 1; break; }
        mbar_expect_tx(&bars->v_full[s], TILE_BYTES);
        load_tile(sm.v[s], &p.map_v, &bars->v_full[s], hk * HD, j * TK, b);
      }
      if (*abort_flag) {
        mbar_wait(&bars->q_full, 0);
        drain_ring<2>(bars->k_full, j + key_ahead);
        drain_ring<2>(bars->v_full, j);
      }
    }
  } else if (warp == 9) {
    if (elect_one()) {
      constexpr uint32_t idesc_qk = attn_idesc<F16>(0);
      constexpr uint32_t idesc_pv = attn_idesc<F16>(1);
      const uint32_t q_addr = smem_u32(sm.q);
      auto issue_s = [&](int j) {
        const int s = j & 1;
        if (!mbar_wait(&bars->k_full[s], (j >> 1) & 1)) return false;
        tc_fence_after();
        const uint32_t k_addr = smem_u32(sm.k[s]);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16_ss(tmem + s * 128, desc_kmajor(q_addr, ks), desc_kmajor(k_addr, ks), idesc_qk, ks != 0);
        umma_commit(&bars->k_empty[s]);
        umma_commit(&bars->s_full[s]);
        return true;
      };
      bool ok = mbar_wait(&bars->q_full, 0) && issue_s(0) && (n_kv < 2 || issue_s(1));
      if (!ok) ATTN_FAIL(203);
      for (int j = 0; j < n_kv && ok && !*abort_flag; ++j) {
        const int s = j & 1;
        if (!mbar_wait(&bars->p_full[s], (j >> 1) & 1) || !mbar_wait(&bars->v_full[s], (j >> 1) & 1)) {
          ATTN_FAIL(205);
          break;
        }
        tc_fence_after();
        const uint32_t v_addr = smem_u32(sm.v[s]);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16_ts(t_o, tmem + s * 128 + (ks >> 2) * 64 + (ks & 3) * 8, desc_mnmajor(v_addr, ks), idesc_pv,
                       (j | ks) != 0);
        umma_commit(&bars->v_empty[s]);
        umma_commit(&bars->o_done);
        if (j + 2 < n_kv && !issue_s(j + 2)) { ATTN_FAIL(204); break; }     // behind the product that reads its P
      }
    }
  } else {
    const int half = warp >> 2;                           // which 64 key columns this thread handles
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                       // query row inside the tile
    const int col0 = half * 64;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t to = t_o + lane_base + col0;
    float m_ref = -INFINITY, l = 0.f;
    for (int j = 0; j < n_kv && !*abort_flag; ++j) {
      const int s = j & 1;
      if (!mbar_wait(&bars->s_full[s], (j >> 1) & 1)) { ATTN_FAIL(206); break; }
      tc_fence_after();
      const uint32_t ts = tmem + s * 128 + lane_base + col0;
      uint32_t raw[2][32];
      tmem_ld_32x32(ts, raw[0]);
      tmem_ld_32x32(ts + 32, raw[1]);
      tmem_ld_wait();
      // keys that the row does not see: after the query (causal, diagonal tile) or behind the sequence
      const bool diagonal = p.causal && j == qt;
      if (diagonal || (j + 1) * TK > p.S) {
        const int limit = (diagonal ? r + 1 : p.S - j * TK) - col0;
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i >= limit) raw[i >> 5][i & 31] = 0xff800000u;   // -inf
      }
      float mpart[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 64; i += 2)
        mpart[(i >> 1) & 3] = fmaxf(fmaxf(mpart[(i >> 1) & 3], __uint_as_float(raw[i >> 5][i & 31])),
                                    __uint_as_float(raw[i >> 5][(i & 31) + 1]));
      float mx = fmaxf(fmaxf(mpart[0], mpart[1]), fmaxf(mpart[2], mpart[3]));
      // exchange with the thread that owns the other 64 columns; two buffers, since that thread may be a tile ahead
      sm.row_max[s][half][r] = mx;
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->row_ready);
      if (!mbar_wait(&bars->row_ready, j & 1)) { ATTN_FAIL(209); break; }
      mx = fmaxf(fmaxf(mx, sm.row_max[s][half ^ 1][r]), m_ref);
      const bool need = (mx - m_ref) * p.scale_log2 > 8.f;      // also true on the first tile (m_ref = -inf)
      const bool any = __any_sync(0xffffffffu, need);
      float alpha = 1.f;
      if (any) {
        alpha = ex2((m_ref - mx) * p.scale_log2);               // 0 on the first tile
        m_ref = mx;
        l *= alpha;
      }
      l += probabilities64<F16, 64>(raw[0], raw[1], ts, p.scale_log2, -m_ref * p.scale_log2);
      if (j > 0) {
        if (!mbar_wait(&bars->o_done, (j - 1) & 1)) { ATTN_FAIL(207); break; }
        tc_fence_after();
        if (any) {
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            uint32_t o[32];
            tmem_ld_32x32(to + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32(to + c * 32, o);
          }
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->p_full[s]);
    }
    // epilogue: add the two halves of the row sum, normalise and store this thread's 64 columns
    if (!*abort_flag) {
      sm.row_sum[half][r] = l;
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->row_ready);
      if (!mbar_wait(&bars->row_ready, n_kv & 1)) ATTN_FAIL(210);
      const float sum = sm.row_sum[0][r] + sm.row_sum[1][r], inv = 1.f / sum;
      if (!mbar_wait(&bars->o_done, (n_kv - 1) & 1)) ATTN_FAIL(208);
      tc_fence_after();
      const int pos = qt * TQ + r;
      uint8_t* dst = static_cast<uint8_t*>(p.out) + (((static_cast<size_t>(b) * p.S + pos) * p.Hq + h) * HD + col0) * 2;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(to + c * 32, o);
        tmem_ld_wait();
        if (pos < p.S) store_out32<F16>(dst + c * 64, o, inv);
        __syncwarp();
      }
      if (half == 0 && pos < p.S) p.lse[static_cast<size_t>(work.head) * p.S + pos] = m_ref * p.scale + logf(sum);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ================================================================= backward: row statistics
// stats[head][0][pos] = -lse * log2(e), stats[head][1][pos] = -rowsum(dO * O); -inf and 0 behind the sequence.  Half a
// warp per row (16 bytes a lane), sixteen consecutive positions of one head per block: 64-byte stores.  Memory bound:
// 134 MB in 32 us at 32 heads of 8192 tokens (a warp per row with 8-byte loads: 48 us).
__global__ void __launch_bounds__(256) attn_stats_kernel(const __nv_bfloat16* __restrict__ dout,
                                                         const __nv_bfloat16* __restrict__ out,
                                                         const float* __restrict__ lse, float* __restrict__ stats, int S,
                                                         int Sp, int Hq) {
  chain_begin();
  const int sub = threadIdx.x & 15;
  const int blocks_per_head = Sp / 16;
  const int head = blockIdx.x / blocks_per_head;           // batch * Hq + h
  const int pos = (blockIdx.x - head * blocks_per_head) * 16 + (threadIdx.x >> 4);
  const int b = head / Hq, h = head - b * Hq;
  float sum = 0.f;
  if (pos < S) {
    const size_t base = ((static_cast<size_t>(b) * S + pos) * Hq + h) * HD + sub * 8;
    const uint4 a = *reinterpret_cast<const uint4*>(dout + base);
    const uint4 o = *reinterpret_cast<const uint4*>(out + base);
    const uint32_t av[4] = {a.x, a.y, a.z, a.w}, ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&av[i]));
      const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ov[i]));
      sum += x.x * y.x + x.y * y.y;
    }
  }
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  if (sub == 0) {
    float* row = stats + static_cast<size_t>(head) * 2 * Sp + pos;
    row[0] = pos < S ? -lse[static_cast<size_t>(head) * S + pos] * 1.4426950408889634f : -INFINITY;
    row[Sp] = -sum;
  }
}

// 32 columns (chunk c) of a finished gradient row.
__device__ __forceinline__ void store_grad_chunk(uint32_t (&a)[32], __nv_bfloat16* dst, int pos, float scale,
                                                 const float* rope_cos, const float* rope_sin, int c) {
#pragma unroll
  for (int i = 0; i < 32; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) * scale);
  if (rope_cos) unrotate32(a, rope_cos, rope_sin, pos, c * 16);
  uint4* d4 = reinterpret_cast<uint4*>(dst + c * 32);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    d4[i] = make_uint4(pack_bf16(__uint_as_float(a[8 * i]), __uint_as_float(a[8 * i + 1])),
                       pack_bf16(__uint_as_float(a[8 * i + 2]), __uint_as_float(a[8 * i + 3])),
                       pack_bf16(__uint_as_float(a[8 * i + 4]), __uint_as_float(a[8 * i + 5])),
                       pack_bf16(__uint_as_float(a[8 * i + 6]), __uint_as_float(a[8 * i + 7])));
}

// A finished accumulator row of 128 fp32 columns: scaled, rotated back if tables are given, stored as bf16.  The whole
// warp calls it (tcgen05.ld is a warp instruction); rows behind the sequence are not stored.  CHUNKS of 32 columns from
// chunk ``first`` on.
template <int CHUNKS = 4>
__device__ __forceinline__ void store_grad_row(uint32_t taddr, __nv_bfloat16* dst, int pos, int S, float scale,
                                               const float* rope_cos, const float* rope_sin, int first = 0) {
#pragma unroll 1
  for (int c = first; c < first + CHUNKS; ++c) {
    uint32_t a[32];
    tmem_ld_32x32(taddr + c * 32, a);
    tmem_ld_wait();
    if (pos < S) store_grad_chunk(a, dst, pos, scale, rope_cos, rope_sin, c);
    __syncwarp();
  }
}

// ================================================================= backward: dK, dV
// Both backward kernels are bound by the chain MMA -> softmax warps -> MMA of a 128 x 128 tile (of 3500 cycles 1050 on
// the special-function unit and 2050 on the tensor core when the two warpgroups ran in step), so the tile is cut into
// two 64-column halves with their own barriers: half a period apart, one half's exponentials run under the other half's
// products and hand-overs.  32/8 heads of 8192 tokens, causal: dK/dV 1058 -> 932 us, dQ 848 -> 714 us.
struct BwdBars {
  uint64_t fixed_full, a_full[3], a_empty[3], b_full[2], b_empty[2], st_full[2], dpt_full[2], p_ready[2], ds_ready[2],
      acc_done;
};
constexpr int HALF = 64;
template <bool V> struct Constant { static constexpr bool value = V; };

// Shared memory of both kernels: two tiles that stay, a ring of three (read last by the products of the previous
// step), a ring of two, and per ring slot 128 row statistics (dK/dV kernel only).
struct BwdSmem {
  uint8_t fixed[2][TILE_BYTES];
  uint8_t a[3][TILE_BYTES];
  uint8_t b[2][TILE_BYTES];
  float a_stat[3][TQ], b_stat[2][TQ];
  BwdBars bars;
  uint32_t tmem_slot;
  int abort_flag;
};

__device__ __forceinline__ void bwd_init(BwdSmem& sm, int warp) {
  if (threadIdx.x == 0) {
    mbar_init(&sm.bars.fixed_full, 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(&sm.bars.a_full[s], 1);
      mbar_init(&sm.bars.a_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sm.bars.b_full[s], 1);
      mbar_init(&sm.bars.b_empty[s], 1);
      mbar_init(&sm.bars.st_full[s], 1);
      mbar_init(&sm.bars.dpt_full[s], 1);
      mbar_init(&sm.bars.p_ready[s], 4);
      mbar_init(&sm.bars.ds_ready[s], 4);
    }
    mbar_init(&sm.bars.acc_done, 1);
    sm.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(&sm.tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_begin();
}

__device__ __forceinline__ void bwd_exit(BwdSmem& sm, int warp, uint32_t tmem) {
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// In grids that leave most SMs idle a cluster of CTAs shares the steps of one tile (launch_bwd): each sums its part in its own
// tensor memory, each adds up an equal share of the rows, in the order of the parts, and stores it.  The parts meet in the
// rings' shared memory once every CTA of the cluster has used its tiles.
__device__ __forceinline__ int cluster_parts() {
  uint32_t n;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
  return static_cast<int>(n);
}
// [first, first + count) of ``steps`` for this CTA of its cluster.
__device__ __forceinline__ void my_steps(int steps, int parts, int& first, int& count) {
  const int per = (steps + parts - 1) / parts, rank = static_cast<int>(cluster_ctarank());
  first = min(steps, rank * per);
  count = min(steps - first, per);
}
// 32 columns of a thread's accumulator row (or zeros) to the CTA that adds up this row: ``sums`` is there [parts][rows per
// CTA][128] floats, 16-byte units swizzled by row.  Stores to the other CTAs' shared memory need no answer; reading the parts
// from there instead takes a round trip per part.
__device__ __forceinline__ void put_sums(float* sums, int parts, int row, int chunk, const uint32_t (&v)[32]) {
  const int rows = 128 / parts, owner = row / rows;
  const uint32_t dst = mapa_u32(smem_u32(sums + (static_cast<int>(cluster_ctarank()) * rows + row - owner * rows) * 128), owner);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (((chunk * 8 + i) ^ (row & 7)) << 4)),
                 "r"(v[4 * i]), "r"(v[4 * i + 1]), "r"(v[4 * i + 2]), "r"(v[4 * i + 3])
                 : "memory");
}
// The sum of the parts for 32 columns of row ``mine`` of this CTA's share (row ``row`` of the tile).
__device__ __forceinline__ void add_sums(const float* sums, int parts, int mine, int row, int chunk, uint32_t (&v)[32]) {
  for (int part = 0; part < parts; ++part) {
    const float4* const src = reinterpret_cast<const float4*>(sums + (part * (128 / parts) + mine) * 128);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 x = src[(chunk * 8 + i) ^ (row & 7)];
      const float y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) v[4 * i + k] = __float_as_uint(part == 0 ? y[k] : __uint_as_float(v[4 * i + k]) + y[k]);
    }
  }
}
// 32 columns of a warp's accumulator rows out of tensor memory, zeros where this CTA had no step.
__device__ __forceinline__ void take_sums(uint32_t taddr, bool here, uint32_t (&v)[32]) {
  if (here) {
    tmem_ld_32x32(taddr, v);
    tmem_ld_wait();
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0;
  }
}

// Slot and phase of step i in a ring of three.
__device__ __forceinline__ int slot3(int i) { return i % 3; }
__device__ __forceinline__ uint32_t phase3(int i) { return (i / 3) & 1; }

__device__ __forceinline__ void arrive_half(uint64_t* bar, int lane) {
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// TMEM: S^T / P^T [0,128), dP^T / dS^T [128,256) (64 columns per half), dV [256,384), dK [384,512).  320 threads: warps
// 0-7 two softmax warpgroups, group g handles query columns [64 g, 64 g + 64) of every tile; warp 8 TMA, warp 9 MMA.
// The ring of three holds Q tiles (with -rowsum(dO O)), the ring of two dO tiles (with -lse).  MMA order per query tile:
//   dV0(i) S0(i+1) | dK1(i-1) dP1(i) | dV1(i) S1(i+1) | dK0(i) dP0(i+1)
// each group of products waits for one half's P or dS, which the other half's turn has given time to appear.
__global__ void __launch_bounds__(ATTN_THREADS, 1) attn_bwd_dkv_kernel(const __grid_constant__ AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  BwdSmem& sm = *reinterpret_cast<BwdSmem*>(smem_raw);
  BwdBars* bars = &sm.bars;
  volatile int* abort_flag = &sm.abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q_tiles = (p.S + TQ - 1) / TQ;
  const int parts = cluster_parts();
  const AttnWork work = attn_work(p, q_tiles, p.B * p.Hkv, static_cast<int>(blockIdx.x) / parts);
  const int kt = work.tile, b = work.head / p.Hkv, hk = work.head - b * p.Hkv;
  const int group = p.Hq / p.Hkv;
  const int q_first = p.causal ? kt : 0;           // causal: query tiles kt .. q_tiles-1
  const int per_head = q_tiles - q_first;
  int it0, iters;                                  // this CTA's steps (query tiles of the group's heads)
  my_steps(group * per_head, parts, it0, iters);

  bwd_init(sm, warp);
  const uint32_t tmem = sm.tmem_slot;
  const uint32_t t_st = tmem, t_dpt = tmem + 128, t_dv = tmem + 256, t_dk = tmem + 384;

  if (warp == 8) {
    if (iters > 0 && elect_one()) {
      mbar_expect_tx(&bars->fixed_full, 2 * TILE_BYTES);
      load_tile(sm.fixed[0], &p.map_k, &bars->fixed_full, hk * HD, kt * TK, b);
      load_tile(sm.fixed[1], &p.map_v, &bars->fixed_full, hk * HD, kt * TK, b);
      int it = 0, a_ahead = 0;
      for (; it < iters && !*abort_flag; ++it) {
        const int s3 = slot3(it), s2 = it & 1;
        const int hq = hk * group + (it0 + it) / per_head;
        const int qi = q_first + (it0 + it) % per_head;
        const float* stat = p.stats + (static_cast<size_t>(b) * p.Hq + hq) * 2 * q_tiles * TQ + qi * TQ;
        if (!mbar_wait(&bars->a_empty[s3], phase3(it) ^ 1)) { ATTN_FAIL(211); break; }
        mbar_expect_tx(&bars->a_full[s3], TILE_BYTES + TQ * 4);
        load_tile(sm.a[s3], &p.map_q, &bars->a_full[s3], hq * HD, qi * TQ, b);
        bulk_load(sm.a_stat[s3], stat + q_tiles * TQ, &bars->a_full[s3], TQ * 4);
        if (!mbar_wait(&bars->b_empty[s2], ((it >> 1) & 1) ^ 1)) { ATTN_FAIL(212); a_ahead = 1; break; }
        mbar_expect_tx(&bars->b_full[s2], TILE_BYTES + TQ * 4);
        load_tile(sm.b[s2], &p.map_do, &bars->b_full[s2], hq * HD, qi * TQ, b);
        bulk_load(sm.b_stat[s2], stat, &bars->b_full[s2], TQ * 4);
      }
      if (*abort_flag) {
        mbar_wait(&bars->fixed_full, 0);
        drain_ring<3>(bars->a_full, it + a_ahead);
        drain_ring<2>(bars->b_full, it);
      }
    }
  } else if (warp == 9) {
    if (iters > 0 && elect_one()) {
      constexpr uint32_t idesc_kk = umma_idesc_bf16(128, HALF, 0, 0);  // both operands K-major
      constexpr uint32_t idesc_tn = umma_idesc_bf16(128, 128, 0, 1);   // A from TMEM, B MN-major
      const uint32_t k_addr = smem_u32(sm.fixed[0]), v_addr = smem_u32(sm.fixed[1]);
      auto issue_st = [&](int it, int g) {          // S^T[key, q half] = K Q^T
        const uint32_t q_addr = smem_u32(sm.a[slot3(it)]) + g * HALF * 128;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16_ss(t_st + g * HALF, desc_kmajor(k_addr, ks), desc_kmajor(q_addr, ks), idesc_kk, ks != 0);
        umma_commit(&bars->st_full[g]);
      };
      auto issue_dpt = [&](int it, int g) {         // dP^T[key, q half] = V dO^T
        const uint32_t do_addr = smem_u32(sm.b[it & 1]) + g * HALF * 128;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16_ss(t_dpt + g * HALF, desc_kmajor(v_addr, ks), desc_kmajor(do_addr, ks), idesc_kk, ks != 0);
        umma_commit(&bars->dpt_full[g]);
      };
      auto issue_dv = [&](int it, int g) {          // dV[key, d] += P^T[key, q half] dO[q half, d]
        const uint32_t do_addr = smem_u32(sm.b[it & 1]);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          umma_bf16_ts(t_dv, t_st + g * HALF + ks * 8, desc_mnmajor(do_addr, g * 4 + ks), idesc_tn, (it | g | ks) != 0);
      };
      auto issue_dk = [&](int it, int g) {          // dK[key, d] += dS^T[key, q half] Q[q half, d]
        const uint32_t q_addr = smem_u32(sm.a[slot3(it)]);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          umma_bf16_ts(t_dk, t_dpt + g * HALF + ks * 8, desc_mnmajor(q_addr, g * 4 + ks), idesc_tn, (it | g | ks) != 0);
      };
      bool ok = mbar_wait(&bars->fixed_full, 0) && mbar_wait(&bars->a_full[0], 0) && mbar_wait(&bars->b_full[0], 0);
      if (ok) {
        tc_fence_after();
        issue_st(0, 0);
        issue_st(0, 1);
        issue_dpt(0, 0);
      }
      for (int it = 0; it < iters && ok && !*abort_flag; ++it) {
        const uint32_t ph = it & 1;
        const bool more = it + 1 < iters;
        if (!(ok = mbar_wait(&bars->p_ready[0], ph))) break;
        tc_fence_after();
        issue_dv(it, 0);
        if (more) {
          if (!(ok = mbar_wait(&bars->a_full[slot3(it + 1)], phase3(it + 1)))) break;
          tc_fence_after();
          issue_st(it + 1, 0);              // overwrites P^T only after dV above (same-thread issue order)
        }
        if (it > 0) {
          if (!(ok = mbar_wait(&bars->ds_ready[1], ph ^ 1))) break;
          tc_fence_after();
          issue_dk(it - 1, 1);
          umma_commit(&bars->a_empty[slot3(it - 1)]);
        }
        issue_dpt(it, 1);                   // overwrites dS^T only after dK above
        if (!(ok = mbar_wait(&bars->p_ready[1], ph))) break;
        tc_fence_after();
        issue_dv(it, 1);
        umma_commit(&bars->b_empty[it & 1]);
        if (more) issue_st(it + 1, 1);
        if (!(ok = mbar_wait(&bars->ds_ready[0], ph))) break;
        tc_fence_after();
        issue_dk(it, 0);
        if (more) {
          if (!(ok = mbar_wait(&bars->b_full[(it + 1) & 1], ((it + 1) >> 1) & 1))) break;
          tc_fence_after();
          issue_dpt(it + 1, 0);
        }
      }
      if (ok && !*abort_flag && (ok = mbar_wait(&bars->ds_ready[1], (iters - 1) & 1))) {
        tc_fence_after();
        issue_dk(iters - 1, 1);
        umma_commit(&bars->acc_done);
      }
      if (!ok) ATTN_FAIL(213);
    }
  } else {
    const int half = warp >> 2;                            // which 64 query columns this thread handles
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                        // key row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const int col0 = half * HALF;
    const uint32_t ts = t_st + lane_base + col0, tp = t_dpt + lane_base + col0;
    const f32x2 scale2 = make_f32x2(p.scale_log2, p.scale_log2);
    for (int it = 0; it < iters && !*abort_flag; ++it) {
      const int qi = q_first + (it0 + it) % per_head;
      const uint32_t ph = it & 1;
      // statistics of my 64 query columns: four columns per 16-byte broadcast read
      const float4* nlse = reinterpret_cast<const float4*>(sm.b_stat[it & 1] + col0);
      const float4* ndelta = reinterpret_cast<const float4*>(sm.a_stat[slot3(it)] + col0);
      if (!mbar_wait(&bars->b_full[it & 1], (it >> 1) & 1) || !mbar_wait(&bars->a_full[slot3(it)], phase3(it)) ||
          !mbar_wait(&bars->st_full[half], ph)) {
        ATTN_FAIL(216);
        break;
      }
      tc_fence_after();
      uint32_t raw[2][32], pk[16];
      f32x2 pf[32];
      tmem_ld_32x32(ts, raw[0]);
      tmem_ld_32x32(ts + 32, raw[1]);
      tmem_ld_wait();
      // P^T as bf16 pairs, written over the first 32 of the 64 columns this thread has just read
      auto probabilities = [&](auto diagonal) {
#pragma unroll
        for (int g = 0; g < 16; ++g) {
          const float4 n = nlse[g];
          const uint32_t* x = &raw[g >> 3][(g & 7) * 4];
          float e[4];
          split_f32x2(fma_f32x2(bits_f32x2(x), scale2, make_f32x2(n.x, n.y)), e[0], e[1]);
          split_f32x2(fma_f32x2(bits_f32x2(x + 2), scale2, make_f32x2(n.z, n.w)), e[2], e[3]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            e[i] = ex2(e[i]);
            if (decltype(diagonal)::value && r > col0 + g * 4 + i) e[i] = 0.f;   // key after query
          }
          pf[2 * g] = make_f32x2(e[0], e[1]);
          pf[2 * g + 1] = make_f32x2(e[2], e[3]);
          pk[(2 * g) & 15] = pack_bf16(e[0], e[1]);
          pk[(2 * g + 1) & 15] = pack_bf16(e[2], e[3]);
          if ((g & 7) == 7) tmem_st_32x16(ts + (g >> 3) * 16, pk);
        }
      };
      if (p.causal && qi == kt) probabilities(Constant<true>());
      else probabilities(Constant<false>());
      tmem_st_wait();
      arrive_half(&bars->p_ready[half], lane);
      if (!mbar_wait(&bars->dpt_full[half], ph)) { ATTN_FAIL(217); break; }
      tc_fence_after();
      tmem_ld_32x32(tp, raw[0]);
      tmem_ld_32x32(tp + 32, raw[1]);
      tmem_ld_wait();
      // dS without the factor 1/sqrt(head_dim), which the epilogue applies to the fp32 sum
#pragma unroll
      for (int g = 0; g < 16; ++g) {
        const float4 n = ndelta[g];
        const uint32_t* x = &raw[g >> 3][(g & 7) * 4];
        float e[4];
        split_f32x2(mul_f32x2(pf[2 * g], add_f32x2(bits_f32x2(x), make_f32x2(n.x, n.y))), e[0], e[1]);
        split_f32x2(mul_f32x2(pf[2 * g + 1], add_f32x2(bits_f32x2(x + 2), make_f32x2(n.z, n.w))), e[2], e[3]);
        pk[(2 * g) & 15] = pack_bf16(e[0], e[1]);
        pk[(2 * g + 1) & 15] = pack_bf16(e[2], e[3]);
        if ((g & 7) == 7) tmem_st_32x16(tp + (g >> 3) * 16, pk);
      }
      tmem_st_wait();
      arrive_half(&bars->ds_ready[half], lane);
    }
    // epilogue: group 0 stores dV, group 1 dK
    if (!*abort_flag && iters > 0 && !mbar_wait(&bars->acc_done, 0)) ATTN_FAIL(218);
    if (parts == 1 && !*abort_flag) {
      tc_fence_after();
      const int pos = kt * TK + r;
      const size_t token = static_cast<size_t>(b) * p.S + pos;
      __nv_bfloat16* dst = half ? p.dk + token * p.dk_pitch + hk * HD : p.dv + token * p.dv_pitch + hk * HD;
      store_grad_row(half ? t_dk + lane_base : t_dv + lane_base, dst, pos, p.S, half ? p.scale : 1.f,
                     half ? p.rope_cos : nullptr, p.rope_sin);
    }
  }
  if (parts > 1) {
    float* const sums = reinterpret_cast<float*>(sm.a);
    __syncwarp();
    cluster_sync_all();                            // every CTA of the cluster has used its tiles
    if (warp < 8) {                                // group 0 hands over dV, group 1 dK
      const int half = warp >> 2;
      const bool here = __all_sync(0xffffffffu, iters > 0 && !*abort_flag);
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        take_sums((half ? t_dk : t_dv) + (static_cast<uint32_t>((warp & 3) * 32) << 16) + c * 32, here, v);
        put_sums(sums + half * 128 * 128, parts, (warp & 3) * 32 + lane, c, v);
      }
    }
    __syncwarp();
    cluster_sync_all();
    const int rows = TK / parts, first = static_cast<int>(cluster_ctarank()) * rows;
#pragma unroll 1
    for (int item = threadIdx.x; item < rows * 8; item += ATTN_THREADS) {
      const int row = first + (item >> 3), which = (item >> 2) & 1, c = item & 3, pos = kt * TK + row;
      if (pos >= p.S || *abort_flag) continue;
      uint32_t v[32];
      add_sums(sums + which * 128 * 128, parts, item >> 3, row, c, v);
      const size_t token = static_cast<size_t>(b) * p.S + pos;
      store_grad_chunk(v, which ? p.dk + token * p.dk_pitch + hk * HD : p.dv + token * p.dv_pitch + hk * HD, pos,
                       which ? p.scale : 1.f, which ? p.rope_cos : nullptr, p.rope_sin, c);
    }
  }
  bwd_exit(sm, warp, tmem);
}

// ================================================================= backward: dQ
// TMEM: S [0,128), dP / dS [128,256), dQ [256,384), Q and dO as A operands [384,448) and [448,512).  Thread layout as above with
// query rows: group g handles key columns [64 g, 64 g + 64).  The ring of three holds K tiles, the ring of two V tiles.  P stays in
// registers, so the next
// scores of a half are issued as soon as its warps have read the present ones (p_ready counts that).  MMA order:
//   S0(j+1) | dQ1(j-1) dP1(j) | S1(j+1) | dQ0(j) dP0(j+1)
__global__ void __launch_bounds__(ATTN_THREADS, 1) attn_bwd_dq_kernel(const __grid_constant__ AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  BwdSmem& sm = *reinterpret_cast<BwdSmem*>(smem_raw);
  BwdBars* bars = &sm.bars;
  volatile int* abort_flag = &sm.abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q_tiles = (p.S + TQ - 1) / TQ;
  const int parts = cluster_parts();
  const AttnWork work = attn_work(p, q_tiles, p.B * p.Hq, static_cast<int>(blockIdx.x) / parts);
  const int qt = q_tiles - 1 - work.tile;
  const int b = work.head / p.Hq, h = work.head - b * p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  int j0, n_kv;                                    // this CTA's key tiles
  my_steps(p.causal ? qt + 1 : q_tiles, parts, j0, n_kv);

  bwd_init(sm, warp);
  const uint32_t tmem = sm.tmem_slot;
  const uint32_t t_s = tmem, t_dp = tmem + 128, t_dq = tmem + 256, t_q = tmem + 384, t_do = tmem + 448;

  if (warp == 8) {
    if (n_kv > 0 && elect_one()) {
      mbar_expect_tx(&bars->fixed_full, 2 * TILE_BYTES);
      load_tile(sm.fixed[0], &p.map_q, &bars->fixed_full, h * HD, qt * TQ, b);
      load_tile(sm.fixed[1], &p.map_do, &bars->fixed_full, h * HD, qt * TQ, b);
      int j = 0, a_ahead = 0;
      for (; j < n_kv && !*abort_flag; ++j) {
        const int s3 = slot3(j), s2 = j & 1;
        if (!mbar_wait(&bars->a_empty[s3], phase3(j) ^ 1)) { ATTN_FAIL(221); break; }
        mbar_expect_tx(&bars->a_full[s3], TILE_BYTES);
        load_tile(sm.a[s3], &p.map_k, &bars->a_full[s3], hk * HD, (j0 + j) * TK, b);
        if (!mbar_wait(&bars->b_empty[s2], ((j >> 1) & 1) ^ 1)) { ATTN_FAIL(222); a_ahead = 1; break; }
        mbar_expect_tx(&bars->b_full[s2], TILE_BYTES);
        load_tile(sm.b[s2], &p.map_v, &bars->b_full[s2], hk * HD, (j0 + j) * TK, b);
      }
      if (*abort_flag) {
        mbar_wait(&bars->fixed_full, 0);
        drain_ring<3>(bars->a_full, j + a_ahead);
        drain_ring<2>(bars->b_full, j);
      }
    }
  } else if (warp == 9) {
    if (n_kv > 0 && elect_one()) {
      constexpr uint32_t idesc_kk = umma_idesc_bf16(128, HALF, 0, 0);
      constexpr uint32_t idesc_tn = umma_idesc_bf16(128, 128, 0, 1);
      auto issue_s = [&](int j, int g) {           // S[q, key half] = Q K^T
        const uint32_t k_addr = smem_u32(sm.a[slot3(j)]) + g * HALF * 128;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16_ts(t_s + g * HALF, t_q + ks * 8, desc_kmajor(k_addr, ks), idesc_kk, ks != 0);
        umma_commit(&bars->st_full[g]);
      };
      auto issue_dp = [&](int j, int g) {          // dP[q, key half] = dO V^T
        const uint32_t v_addr = smem_u32(sm.b[j & 1]) + g * HALF * 128;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_bf16_ts(t_dp + g * HALF, t_do + ks * 8, desc_kmajor(v_addr, ks), idesc_kk, ks != 0);
        umma_commit(&bars->dpt_full[g]);
      };
      auto issue_dq = [&](int j, int g) {          // dQ[q, d] += dS[q, key half] K[key half, d]
        const uint32_t k_addr = smem_u32(sm.a[slot3(j)]);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          umma_bf16_ts(t_dq, t_dp + g * HALF + ks * 8, desc_mnmajor(k_addr, g * 4 + ks), idesc_tn, (j | g | ks) != 0);
      };
      // Q and dO are in tensor memory once both groups have copied their tile (see below)
      bool ok = mbar_wait(&bars->ds_ready[0], 0) && mbar_wait(&bars->ds_ready[1], 0) && mbar_wait(&bars->a_full[0], 0) &&
                mbar_wait(&bars->b_full[0], 0);
      if (ok) {
        tc_fence_after();
        issue_s(0, 0);
        issue_s(0, 1);
        issue_dp(0, 0);
      }
      for (int j = 0; j < n_kv && ok && !*abort_flag; ++j) {
        const uint32_t ph = j & 1;
        const bool more = j + 1 < n_kv;
        if (more) {
          if (!(ok = mbar_wait(&bars->a_full[slot3(j + 1)], phase3(j + 1)) && mbar_wait(&bars->p_ready[0], ph))) break;
          tc_fence_after();
          issue_s(j + 1, 0);
        }
        if (j > 0) {
          if (!(ok = mbar_wait(&bars->ds_ready[1], ph))) break;
          tc_fence_after();
          issue_dq(j - 1, 1);
          umma_commit(&bars->a_empty[slot3(j - 1)]);
        }
        issue_dp(j, 1);                     // overwrites dS only after dQ above
        umma_commit(&bars->b_empty[j & 1]);
        if (more) {
          if (!(ok = mbar_wait(&bars->p_ready[1], ph))) break;
          tc_fence_after();
          issue_s(j + 1, 1);
        }
        if (!(ok = mbar_wait(&bars->ds_ready[0], ph ^ 1))) break;
        tc_fence_after();
        issue_dq(j, 0);
        if (more) {
          if (!(ok = mbar_wait(&bars->b_full[(j + 1) & 1], ((j + 1) >> 1) & 1))) break;
          tc_fence_after();
          issue_dp(j + 1, 0);
        }
      }
      if (ok && !*abort_flag && (ok = mbar_wait(&bars->ds_ready[1], n_kv & 1))) {
        tc_fence_after();
        issue_dq(n_kv - 1, 1);
        umma_commit(&bars->acc_done);
      }
      if (!ok) ATTN_FAIL(223);
    }
  } else {
    const int half = warp >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                        // query row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const int col0 = half * HALF;
    const uint32_t ts = t_s + lane_base + col0, tp = t_dp + lane_base + col0;
    const float* stat = p.stats + static_cast<size_t>(work.head) * 2 * q_tiles * TQ + qt * TQ + r;
    const f32x2 scale2 = make_f32x2(p.scale_log2, p.scale_log2);
    const f32x2 nlse2 = make_f32x2(stat[0], stat[0]);
    const f32x2 ndelta2 = make_f32x2(stat[q_tiles * TQ], stat[q_tiles * TQ]);
    // The A operands of both score products, the same for every key tile, move to tensor memory: group 0 copies Q, group 1
    // dO, a row per thread (16-byte units of the 128-byte-swizzled tile).  From shared memory they were read again for every
    // 64 keys, and the products with N = 64 waited for it (6 KiB per 32 cycles): 32/8 heads of 8192 tokens, causal, backward
    // pass as a whole 1609 -> 1546 us, 128 heads of 640 tokens, every key, 158 -> 153.
    if (n_kv > 0 && !mbar_wait(&bars->fixed_full, 0)) ATTN_FAIL(224);
    if (n_kv > 0 && !*abort_flag) {
      const uint8_t* row = sm.fixed[half] + r * 128;
#pragma unroll
      for (int atom = 0; atom < 2; ++atom) {
        uint32_t w[32];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint4 x = *reinterpret_cast<const uint4*>(row + atom * ATOM_BYTES + ((u ^ (r & 7)) << 4));
          w[4 * u] = x.x; w[4 * u + 1] = x.y; w[4 * u + 2] = x.z; w[4 * u + 3] = x.w;
        }
        tmem_st_32x32((half ? t_do : t_q) + lane_base + atom * 32, w);
      }
      tmem_st_wait();
      arrive_half(&bars->ds_ready[half], lane);
    }
    for (int j = 0; j < n_kv && !*abort_flag; ++j) {
      const uint32_t ph = j & 1;
      if (!mbar_wait(&bars->st_full[half], ph)) { ATTN_FAIL(225); break; }
      tc_fence_after();
      uint32_t raw[2][32];
      f32x2 pf[32];
      tmem_ld_32x32(ts, raw[0]);
      tmem_ld_32x32(ts + 32, raw[1]);
      tmem_ld_wait();
      arrive_half(&bars->p_ready[half], lane);
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        float e0, e1;
        split_f32x2(fma_f32x2(bits_f32x2(&raw[i >> 4][(i & 15) * 2]), scale2, nlse2), e0, e1);
        pf[i] = make_f32x2(ex2(e0), ex2(e1));
      }
      // keys that the row does not see: after the query (causal, diagonal tile) or behind the sequence
      const bool diagonal = p.causal && j0 + j == qt;
      if (diagonal || (j0 + j + 1) * TK > p.S) {
        const int limit = (diagonal ? r + 1 : p.S - (j0 + j) * TK) - col0;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          float e0, e1;
          split_f32x2(pf[i], e0, e1);
          pf[i] = make_f32x2(2 * i < limit ? e0 : 0.f, 2 * i + 1 < limit ? e1 : 0.f);
        }
      }
      if (!mbar_wait(&bars->dpt_full[half], ph)) { ATTN_FAIL(226); break; }
      tc_fence_after();
      uint32_t pk[32];
      tmem_ld_32x32(tp, raw[0]);
      tmem_ld_32x32(tp + 32, raw[1]);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) {      // dS without the factor 1/sqrt(head_dim): the epilogue applies it
        float e0, e1;
        split_f32x2(mul_f32x2(pf[i], add_f32x2(bits_f32x2(&raw[i >> 4][(i & 15) * 2]), ndelta2)), e0, e1);
        pk[i] = pack_bf16(e0, e1);
      }
      tmem_st_32x32(tp, pk);              // dS pairs over the columns just read
      tmem_st_wait();
      arrive_half(&bars->ds_ready[half], lane);
    }
    if (!*abort_flag && n_kv > 0 && !mbar_wait(&bars->acc_done, 0)) ATTN_FAIL(227);
    if (parts == 1 && !*abort_flag) {     // each group stores 64 of the 128 columns
      tc_fence_after();
      const int pos = qt * TQ + r;
      store_grad_row<2>(t_dq + lane_base, p.dq + (static_cast<size_t>(b) * p.S + pos) * p.dq_pitch + h * HD, pos, p.S,
                        p.scale, p.rope_cos, p.rope_sin, 2 * half);
    }
  }
  if (parts > 1) {
    float* const sums = reinterpret_cast<float*>(sm.a);
    __syncwarp();
    cluster_sync_all();
    if (warp < 8) {                                // each group hands over 64 columns
      const int half = warp >> 2;
      const bool here = __all_sync(0xffffffffu, n_kv > 0 && !*abort_flag);
      tc_fence_after();
#pragma unroll 1
      for (int c = 2 * half; c < 2 * half + 2; ++c) {
        uint32_t v[32];
        take_sums(t_dq + (static_cast<uint32_t>((warp & 3) * 32) << 16) + c * 32, here, v);
        put_sums(sums, parts, (warp & 3) * 32 + lane, c, v);
      }
    }
    __syncwarp();
    cluster_sync_all();
    const int rows = TQ / parts, first = static_cast<int>(cluster_ctarank()) * rows;
#pragma unroll 1
    for (int item = threadIdx.x; item < rows * 4; item += ATTN_THREADS) {
      const int row = first + (item >> 2), c = item & 3, pos = qt * TQ + row;
      if (pos >= p.S || *abort_flag) continue;
      uint32_t v[32];
      add_sums(sums, parts, item >> 2, row, c, v);
      store_grad_chunk(v, p.dq + (static_cast<size_t>(b) * p.S + pos) * p.dq_pitch + h * HD, pos, p.scale, p.rope_cos,
                       p.rope_sin, c);
    }
  }
  bwd_exit(sm, warp, tmem);
}

// ================================================================= host
// [B, S, heads*128] 16-bit elements with token pitch ``pitch`` elements; box = 128 tokens x 64 columns of one batch
// entry (tokens behind the sequence are out of bounds, so they read as zeros instead of the next entry's rows).
static int g_last_encode_result = 0;     // CUresult of the last tensor-map encode that failed (diagnostics)

static int attn_map(CUtensorMap* map, const void* base, int B, int S, int heads, long long pitch, bool f16 = false) {
  EncodeTiledFn fn = encode_fn();      // binds this thread's context first (tensormap.cuh)
  if (!fn) return -1;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(heads) * HD, static_cast<cuuint64_t>(S), static_cast<cuuint64_t>(B)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(pitch) * 2, static_cast<cuuint64_t>(pitch) * 2 * S};
  cuuint32_t box[3] = {64, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult rc = fn(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) g_last_encode_result = static_cast<int>(rc);
  return rc == CUDA_SUCCESS ? 0 : -2;
}

// Heads per launch-order set: as many as keep the tensors that their CTAs read again and again (``bytes_per_head``)
// inside 48 MB of the 126 MB L2; the longest tiles of the whole set start first.
static int heads_per_set(int heads, long long bytes_per_head) {
  const long long fit = (48LL << 20) / (bytes_per_head > 0 ? bytes_per_head : 1);
  return static_cast<int>(fit < 1 ? 1 : (fit > heads ? heads : fit));
}

// The dynamic windows start 1024-byte aligned (the kernels have no static shared memory).
constexpr int FWD_SMEM = 6 * TILE_BYTES + 512;
constexpr int FWD_ONE_SMEM = sizeof(FwdOneSmem);
constexpr int BWD_SMEM = sizeof(BwdSmem);
static_assert(BWD_SMEM <= 227 * 1024, "shared memory of a backward CTA");

static int sm_count_attn() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      sms = 0;
  }
  return sms > 0 ? sms : 148;
}

// Clusters of ``parts`` (2 or 4) backward CTAs that the device holds at once; a cluster lies in one GPC, so that 148 SMs hold 74 of
// two and 33 of four.  Asked once per device.
template <void (*kernel)(AttnParams)>
static int bwd_clusters_resident(int parts) {
  constexpr int DEVICES = 64;
  static std::atomic<int> known[DEVICES][2];                            // 0: not asked yet, else the number + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= DEVICES) return 0;
  std::atomic<int>& slot = known[dev][parts == 4];
  if (slot.load() == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = parts;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(parts);
    cfg.blockDim = dim3(ATTN_THREADS);
    cfg.dynamicSmemBytes = BWD_SMEM;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int count = 0;
    if (cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      count = 0;
    }
    slot.store(count + 1);
  }
  return slot.load() - 1;
}

// A backward kernel over ``tiles`` tiles of at most ``steps`` steps each.  Where the clusters of several parts per tile make one
// wave, two share the steps from seven on and four from eight on: below, the two barriers and the exchange cost what the steps
// save (two parts against one: five steps 29.0, 25.0; six 29.5, 27.5); eight parts gain nothing more.  One wave is what the
// device holds in clusters, 33 of four CTAs, not 148 / 4: 36 tiles of nine steps in four parts are 61 us, in two 35, in one 39.
// Causal tiles of many steps may make a second wave, which the shortest of them fill: 36 tiles of up to 36 steps in four parts
// 53, in two 59.  us, whole backward pass, one -> several parts, causal: 2 x 512 tokens, 4/1 heads 45.8 -> 34.0; 1024, 8/2 73.3 ->
// 41.2; 2048, 8/2 130 -> 68.7; 4 x 1024, 8/2 88.8 -> 70.6; 128, 8/2 (one part) 26.1.
template <void (*kernel)(AttnParams)>
static int launch_bwd(long long tiles, long long steps, const AttnParams& p, cudaStream_t stream) {
  const int sms = sm_count_attn();
  int parts = 1;
  if (steps >= 7 && tiles * 2 <= sms && tiles <= bwd_clusters_resident<kernel>(2)) parts = 2;
  if (steps >= 8 && tiles * 4 <= sms) {
    const int held = bwd_clusters_resident<kernel>(4);
    if (tiles <= held || (held > 0 && p.causal && steps >= 24)) parts = 4;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // chain.cuh
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = parts;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * parts));
  cfg.blockDim = dim3(ATTN_THREADS);
  cfg.dynamicSmemBytes = BWD_SMEM;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = parts > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, p) == cudaSuccess) return 0;
  cudaGetLastError();                                                   // not the next launch's
  return -4;
}

template <void (*kernel)(AttnParams), int smem, int threads = ATTN_THREADS>
static int launch_fwd(const AttnParams& p, long long ctas, cudaStream_t stream) {
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -3;
    set = true;
  }
  launch_next(kernel, static_cast<unsigned>(ctas), threads, smem, stream, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace b2

using namespace b2;

extern "C" {

// After an entry point returned -11 (a tensor map could not be encoded): the driver's result code of that encode.
int b2_attention_last_encode_result() { return g_last_encode_result; }

// q: [B,S,Hq,128], k, v: [B,S,Hkv,128] with token pitches (elements), bf16 or (f16 != 0) fp16; out [B,S,Hq,128]
// contiguous in the same type; lse [B,Hq,S].
int b2_attention_fwd_ex(const void* q, const void* k, const void* v, long long q_pitch, long long k_pitch,
                        long long v_pitch, void* out, float* lse, int B, int S, int Hq, int Hkv, float scale,
                        int causal, int f16, int* status, cudaStream_t stream) {
  if (S < 1 || B < 1 || Hkv < 1 || Hq % Hkv || q_pitch % 8 || k_pitch % 8 || v_pitch % 8) return -10;
  AttnParams p{};
  if (attn_map(&p.map_q, q, B, S, Hq, q_pitch, f16 != 0)) return -11;
  if (attn_map(&p.map_k, k, B, S, Hkv, k_pitch, f16 != 0)) return -12;
  if (attn_map(&p.map_v, v, B, S, Hkv, v_pitch, f16 != 0)) return -13;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv; p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal != 0;
  p.set_heads = heads_per_set(B * Hq, 4LL * S * HD * Hkv / Hq);
  p.out = out; p.lse = lse; p.status = status;
  const long long tiles = (S + TQ - 1) / TQ;
  const long long heads = static_cast<long long>(B) * Hq;
  if (tiles * heads > 0x7fffffffLL) return -10;
  // one wave of one-tile CTAs, or heads of a single tile (nothing to ping-pong with): see attn_fwd_one_tile_kernel
  if (tiles == 1 || tiles * heads <= sm_count_attn())
    return f16 ? launch_fwd<attn_fwd_one_tile_kernel<1>, FWD_ONE_SMEM>(p, tiles * heads, stream)
               : launch_fwd<attn_fwd_one_tile_kernel<0>, FWD_ONE_SMEM>(p, tiles * heads, stream);
  const long long ctas = (tiles + 1) / 2 * heads;
  return f16 ? launch_fwd<attn_fwd_kernel<1>, FWD_SMEM, FWD_THREADS>(p, ctas, stream)
             : launch_fwd<attn_fwd_kernel<0>, FWD_SMEM, FWD_THREADS>(p, ctas, stream);
}

// Gradients.  dout, out: [B,S,Hq,128] contiguous; stats: fp32 scratch [B*Hq, 2, Sp] with Sp = S rounded up to 128; dq
// [B,S,Hq,128], dk, dv [B,S,Hkv,128] with token pitches dq_pitch, dk_pitch, dv_pitch (they may be views into one fused
// gradient buffer).  With rotary tables (fp32 [S, 64]) q and k are the ROTATED tensors the forward pass saw, and dq, dk
// are stored rotated back, i.e. as gradients of the unrotated projections.
int b2_attention_bwd_rope(const void* dout, const void* q, const void* k, const void* v, const void* out,
                          const float* lse, long long q_pitch, long long k_pitch, long long v_pitch, float* stats,
                          void* dq, void* dk, void* dv, long long dq_pitch, long long dk_pitch, long long dv_pitch,
                          int B, int S, int Hq, int Hkv, float scale, int causal, const float* rope_cos,
                          const float* rope_sin, int* status, cudaStream_t stream) {
  if (S < 1 || B < 1 || Hkv < 1 || Hq % Hkv) return -10;
  AttnParams p{};
  // -11 / -12 / -13 / -14: the tensor map of q / k / v / dout could not be encoded (base not 16-byte aligned, pitch
  // not a multiple of 8 elements, ...); b2_attention_last_encode_result() has the driver's code
  if (q_pitch % 8 || k_pitch % 8 || v_pitch % 8) return -10;
  if (attn_map(&p.map_q, q, B, S, Hq, q_pitch)) return -11;
  if (attn_map(&p.map_k, k, B, S, Hkv, k_pitch)) return -12;
  if (attn_map(&p.map_v, v, B, S, Hkv, v_pitch)) return -13;
  if (attn_map(&p.map_do, dout, B, S, Hq, static_cast<long long>(Hq) * HD)) return -14;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv; p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal != 0;
  p.stats = stats; p.dq = static_cast<__nv_bfloat16*>(dq);
  p.dk = static_cast<__nv_bfloat16*>(dk); p.dv = static_cast<__nv_bfloat16*>(dv); p.status = status;
  p.dq_pitch = dq_pitch; p.dk_pitch = dk_pitch; p.dv_pitch = dv_pitch;
  p.rope_cos = rope_cos; p.rope_sin = rope_sin;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(attn_bwd_dkv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(attn_bwd_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM) != cudaSuccess)
      return -3;
    set = true;
  }
  const long long tiles = (S + TQ - 1) / TQ, Sp = tiles * TQ;
  if (Sp / 16 * B * Hq > 0x7fffffffLL) return -10;
  launch_next(attn_stats_kernel, static_cast<unsigned>(Sp / 16 * B * Hq), 256, 0, stream, static_cast<const __nv_bfloat16*>(dout),
              static_cast<const __nv_bfloat16*>(out), lse, stats, S, static_cast<int>(Sp), Hq);
  p.set_heads = heads_per_set(B * Hkv, 4LL * S * HD * (Hq / Hkv));
  if (launch_bwd<attn_bwd_dkv_kernel>(tiles * B * Hkv, tiles * (Hq / Hkv), p, stream)) return -4;
  p.set_heads = heads_per_set(B * Hq, 4LL * S * HD * Hkv / Hq);
  if (launch_bwd<attn_bwd_dq_kernel>(tiles * B * Hq, tiles, p, stream)) return -4;
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // extern "C"
