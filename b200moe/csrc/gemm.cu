// bf16 GEMM family on 5th-generation tensor cores (tcgen05), fp32 accumulation in
// tensor memory, operands staged by TMA (one plain tile load per CTA and tile).
//
// One persistent kernel template covers every contraction of the training step:
//   NT  y = x W^T            (forward linears, grouped expert forward)
//   NN  dx = dy W            (data gradients; W is read MN-major, no transpose copy)
//   TN  dW (+)= dy^T x       (weight gradients, accumulated in fp32 or bf16 in place)
// with a device-side tile table for grouped (per-expert) problems, a fused
// SwiGLU epilogue for the gate/up projection and a K-concatenated form for
// dx = dgate W1 + dup W3.
//
// Layout of one CTA (320 threads, one CTA per SM):
//   warp 0       TMA producer (one elected lane)
//   warp 1       tensor-memory allocation, MMA issue (one elected lane)
//   warps 2..9   epilogue: tcgen05.ld the 128 x BN fp32 tile, convert, store
// The accumulator is double-buffered in TMEM (2 x 256 columns), so the epilogue
// of tile i overlaps the main loop of tile i+1.  Shared memory holds a 4-stage
// ring of {A 128x64, B 256x64} bf16 tiles in the 128-byte-swizzled layout that
// both TMA and the MMA descriptors understand.
#include "chain.cuh"
#include "entries.h"
#include "peer.cuh"
#include "ptx.cuh"
#include "tensormap.cuh"

namespace b2 {

constexpr int BM = 128;
constexpr int BN = 256;                    // columns of a tile; 128 and 64 for small products (``NT`` below)
constexpr int BK = 64;
constexpr int A_SUB_BYTES = BM * BK * 2;   // 16 KiB per 128-row sub-tile of A
// MT = 128-row sub-tiles of A per CTA tile.  MT=1: 128x256 tile, 4 stages, accumulator double-buffered in
// TMEM (epilogue overlaps the next main loop).  MT=2: 256x256 tile (two MMAs per k-step share the B tile in
// shared memory, a third fewer operand bytes per FLOP), 3 stages, both accumulators fill TMEM.
// PAIR = 1 (with MT = 1): two CTAs of a cluster share a 256x256 tile (tcgen05 cta_group::2).  Each CTA stages its
// own 128 rows of A and 128 rows/columns of B (32 KiB per stage, 6 stages), the even CTA issues the MMAs for both,
// and each CTA's tensor memory holds its 128 rows x 256 columns, double-buffered: the operand traffic of a 256x256
// tile with the epilogue overlap of a 128x256 one.
// NT = columns of the tile.  128 and 64 (MT = 1, no pair) are for products whose 128x256 tiles leave SMs without work.
template <int MT, int PAIR = 0, int NT = BN> struct Cfg {
  static constexpr int STAGES = PAIR ? 6 : MT == 2 ? 3 : NT == 256 ? 4 : NT == 128 ? 6 : 8;
  static constexpr int A_BYTES = MT * A_SUB_BYTES;
  static constexpr int B_BYTES = NT * BK * 2;
  static constexpr int B_STAGE_BYTES = PAIR ? B_BYTES / 2 : B_BYTES;
  static constexpr int STAGE_BYTES = A_BYTES + B_STAGE_BYTES;
  static constexpr int NACC = MT == 2 ? 1 : 2;
  static constexpr int TM = PAIR ? 2 : MT;     // 128-row units per output tile
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};
// Epilogue: eight warps, each 32 rows of one half of the tile's columns, through 4 KiB of shared memory per warp (see
// ``staged`` below).  EPI_PUSH: four warps with 8 KiB each, so that a row leaves in pieces of 256 bytes.
constexpr int EPI_STAGING = 32 * 1024;
template <int EPI> constexpr int epi_warps() { return EPI == 5 /*EPI_PUSH*/ ? 4 : 8; }
template <int EPI> constexpr int gemm_threads() { return 64 + 32 * epi_warps<EPI>(); }
template <int EPI, int MT, int PAIR = 0, int NT = BN> constexpr int smem_bytes() { return Cfg<MT, PAIR, NT>::SMEM + EPI_STAGING; }
constexpr int GROUP_M = 8;

enum Epilogue : int {
  EPI_STORE_BF16 = 0,   // D[M,N] bf16 = acc
  EPI_ACC_F32 = 1,      // D[M,N] fp32 += acc   (beta selects += or =)
  EPI_ACC_BF16 = 2,     // D[M,N] bf16 += acc
  EPI_SWIGLU = 3,       // H[M,N/2] = silu(acc[:, :128]) * acc[:, 128:]; optional gate/up stores
  EPI_STORE_F32 = 4,    // D[M,N] fp32 = acc
  EPI_ROPE = 6,         // D[M,N] bf16 = acc with the rotary embedding applied to the leading rope_cols columns
                        // (adjacent pairs, heads of 128 columns, position = row mod rope_seq): the fused q/k/v projection
  EPI_SWIGLU_BWD = 7,   // acc = dh; with the saved pre-activations g, u of the same element: D[M,2N] = [dg | du], H[M,N] =
                        // silu(g) u.  Memory traffic of the epilogue: 2 reads and 3 writes of 2 bytes per element, under
                        // the next tile's main loop; a kernel of its own moved 6 and the GEMM's store of dh a seventh
  EPI_PUSH = 5,         // expert-parallel return: row r, scaled by push_w[r], is stored as bf16 into row push_tag[r]
                        // of rank push_src[r]'s buffer through its peer pointer; the last CTA raises a flag
};

enum Schedule : int {
  SCHED_FLAT = 0,       // tiles over (M, N); optional per-m-tile expert for B
  SCHED_WGRAD = 1,      // tiles over (expert, M, N); K range = rows of the expert
};

struct GemmParams {
  CUtensorMap map_a;
  CUtensorMap map_b;
  CUtensorMap map_d, map_d2;   // fp32 results: d, d2 as the epilogue's bulk stores address them
  CUtensorMap map_b2;          // second B: up-projection (SwiGLU) or K-continuation (k >= k_split)
  int M, N, K;                 // problem per expert for SCHED_WGRAD (K unused there)
  int num_experts;             // >= 1
  int b_expert_rows;           // rows of one expert in the B map (outer TMA coordinate pitch)
  int k_split;                 // K index where map_b2 takes over (0 = unused)
  const int* tile_expert;      // [m_tiles] expert of each m-tile, or null
  const int* num_m_tiles;      // device scalar: live 128-row tiles, or null (= ceil(M/128))
  int group_align256;          // grouped problems: every expert segment is a multiple of 256 rows
  const int* expert_offsets;   // [E] cumulative row ends (SCHED_WGRAD)
  const int* expert_counts;    // optional [E]: rows of each segment that count; the reduction leaves out the zero rows
                               // of its padding (a tenth of 10006 rows in eight segments of whole 256-row tiles)
  void* d;                     // output
  void* d2;                    // optional (EPI_ACC_*): rows from m_split on go to rows [0, M - m_split) of this one
  int m_split;
  void* d_gate;                // optional gate pre-activation (SwiGLU)
  void* d_up;                  // optional up pre-activation (SwiGLU)
  void* h;                     // EPI_SWIGLU_BWD: [M, N]; d_gate and d_up are inputs there
  long long ldd;               // leading dimension of d (elements)
  long long d_expert_stride;   // elements between experts in d (SCHED_WGRAD)
  float beta;                  // 1 accumulate, 0 overwrite (EPI_ACC_*)
  const float* alpha;          // optional device scalar that multiplies the product (EPI_STORE_*, EPI_ACC_*)
  int* status;                 // device word; non-zero = a wait ran out
  // EPI_ROPE only
  const float* rope_cos;       // [rope_seq, 64] fp32
  const float* rope_sin;
  int rope_cols, rope_seq;
  // EPI_PUSH only
  Peers push_dst;              // every rank's return buffer [slots, ldd] bf16
  const int* push_tag;         // [M] destination row (slot id) of each row, -1 for padding rows
  const int* push_src;         // [M] destination rank
  const float* push_w;         // [M] scale (routing weight), or null for 1
  Peers push_sig;              // signal pads
  int push_slot, push_seq, push_rank, push_n;
  unsigned int* push_ticket;   // self-resetting CTA counter
};

struct TileCoord {
  int m_tile, n_tile, expert, k_begin, k_blocks;
  bool valid;
};

template <int SCHED, int MT>
__device__ __forceinline__ TileCoord decode_tile(const GemmParams& p, long long tile, int m_tiles, int n_tiles) {
  TileCoord t;
  t.valid = true;
  if (SCHED == SCHED_WGRAD) {
    const long long per_expert = static_cast<long long>(m_tiles) * n_tiles;
    t.expert = static_cast<int>(tile / per_expert);
    const int rest = static_cast<int>(tile - t.expert * per_expert);
    const int group = rest / (GROUP_M * n_tiles);
    const int first_m = group * GROUP_M;
    const int rows_in_group = min(GROUP_M, m_tiles - first_m);
    const int in_group = rest - group * GROUP_M * n_tiles;
    t.m_tile = first_m + in_group % rows_in_group;
    t.n_tile = in_group / rows_in_group;
    const int begin = t.expert == 0 ? 0 : p.expert_offsets[t.expert - 1];
    const int end = p.expert_counts ? begin + p.expert_counts[t.expert] : p.expert_offsets[t.expert];
    t.k_begin = begin;
    t.k_blocks = (end - begin + BK - 1) / BK;
  } else {
    const int group = static_cast<int>(tile / (GROUP_M * n_tiles));
    const int first_m = group * GROUP_M;
    const int rows_in_group = min(GROUP_M, m_tiles - first_m);
    const int in_group = static_cast<int>(tile - static_cast<long long>(group) * GROUP_M * n_tiles);
    t.m_tile = first_m + in_group % rows_in_group;
    t.n_tile = in_group / rows_in_group;
    t.expert = p.tile_expert ? p.tile_expert[t.m_tile * MT] : 0;
    t.k_begin = 0;
    t.k_blocks = (p.K + BK - 1) / BK;
  }
  return t;
}

template <int A_MN, int B_MN, int EPI, int SCHED, int MT, int PAIR, int NT = BN>
__global__ void __launch_bounds__(gemm_threads<EPI>(), 1) gemm_tcgen05_kernel(const __grid_constant__ GemmParams p) {
  static_assert(!PAIR || MT == 1, "a CTA of a pair holds one 128-row sub-tile");
  static_assert(NT == BN || (MT == 1 && !PAIR && EPI != EPI_PUSH), "narrow tiles: one CTA, 128 rows");
  constexpr int STAGES = Cfg<MT, PAIR, NT>::STAGES;
  constexpr int A_BYTES = Cfg<MT, PAIR, NT>::A_BYTES;
  constexpr int STAGE_BYTES = Cfg<MT, PAIR, NT>::STAGE_BYTES;
  constexpr int NACC = Cfg<MT, PAIR, NT>::NACC;
  constexpr int TM = Cfg<MT, PAIR, NT>::TM;
  constexpr int TILE_M = BM * TM;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES + EPI_STAGING);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full = empty_bar + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // pair mode: ``cta`` is this CTA's half of the tile (0 = leader), a "worker" is a CTA pair
  const uint32_t cta = PAIR ? cluster_ctarank() : 0;
  const int worker = PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int num_workers = PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], (PAIR ? 2 : 1) * epi_warps<EPI>());   // epilogue warps (of both CTAs of a pair)
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.map_a);
    tma_prefetch_desc(&p.map_b);
    if (EPI == EPI_SWIGLU || p.k_split > 0) tma_prefetch_desc(&p.map_b2);
  }
  if (PAIR) {
    __syncthreads();
    cluster_sync_all();      // both CTAs' barriers exist before a remote arrive or a remote completion can reach them
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(tmem_slot, 512);     // one collective allocation by one warp of each CTA
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_begin();
  const int m_tiles = p.num_m_tiles ? (*p.num_m_tiles + TM - 1) / TM : (p.M + TILE_M - 1) / TILE_M;
  const int n_tiles = (p.N + NT - 1) / NT;
  const long long total_tiles = static_cast<long long>(m_tiles) * n_tiles * (SCHED == SCHED_WGRAD ? p.num_experts : 1);

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (every CTA)
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool wrapped = false;       // every stage has been requested at least once
      for (long long tile = worker; tile < total_tiles && !*abort_flag; tile += num_workers) {
        const TileCoord t = decode_tile<SCHED, TM>(p, tile, m_tiles, n_tiles);
        const int m0 = t.m_tile * TILE_M + (PAIR ? static_cast<int>(cta) * BM : 0);
        const int n0 = t.n_tile * NT + (PAIR ? static_cast<int>(cta) * (NT / 2) : 0);
        for (int kb = 0; kb < t.k_blocks; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
            *abort_flag = 1;
            atomicExch(p.status, 1);
            break;
          }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          // pair: the leader's barrier counts the bytes of both CTAs; every load names that barrier
          uint64_t* const full = &full_bar[stage];
          const uint32_t full_on_leader = PAIR ? mapa_u32(smem_u32(full), 0) : 0;
          if (!PAIR) mbar_expect_tx(full, STAGE_BYTES);
          else if (cta == 0) mbar_expect_tx(full, 2 * STAGE_BYTES);
          auto load = [&](void* dst, const CUtensorMap* map, int c0, int c1) {
            if (PAIR) tma_load_2d_pair(dst, map, full_on_leader, c0, c1);
            else tma_load_2d(dst, map, full, c0, c1);
          };
          const int k0 = t.k_begin + kb * BK;
          // ---- A
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            if (A_MN) {
              // MN-major: two boxes of [64 (m) x 64 (k)]; inner coordinate = m, outer = k row
              load(sa + i * A_SUB_BYTES, &p.map_a, m0 + i * BM, k0);
              load(sa + i * A_SUB_BYTES + 8192, &p.map_a, m0 + i * BM + 64, k0);
            } else {
              load(sa + i * A_SUB_BYTES, &p.map_a, k0, m0 + i * BM);
            }
          }
          // ---- B
          if (EPI == EPI_SWIGLU) {
            // gate rows then up rows of the same NT / 2 output features (K-major)
            const int row = t.expert * p.b_expert_rows + t.n_tile * (NT / 2);
            if (PAIR) {
              load(sb, cta == 0 ? &p.map_b : &p.map_b2, k0, row);      // leader: gate rows, peer: up rows
            } else {
              load(sb, &p.map_b, k0, row);
              load(sb + NT * 64, &p.map_b2, k0, row);
            }
          } else if (B_MN) {
            const bool second = p.k_split > 0 && k0 >= p.k_split;
            const CUtensorMap* map = second ? &p.map_b2 : &p.map_b;
            const int krow = (SCHED == SCHED_WGRAD ? 0 : t.expert * p.b_expert_rows) + (second ? k0 - p.k_split : k0);
#pragma unroll
            for (int c = 0; c < (PAIR ? NT / 128 : NT / 64); ++c) load(sb + c * 8192, map, n0 + c * 64, krow);
          } else {
            load(sb, &p.map_b, k0, t.expert * p.b_expert_rows + n0);     // box of NT rows (128 in pair mode)
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
            wrapped = true;
          }
        }
      }
      // a CTA that gives up waits (with a limit) for its copies before its shared memory goes to another one; the
      // leader's barriers count those of both CTAs of a pair
      if (*abort_flag && cta == 0) {
        for (int s = 0; s < STAGES; ++s)
          if (wrapped || s < stage) mbar_wait(&full_bar[s], s < stage ? phase : phase ^ 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the leader of a pair)
    if (cta == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(PAIR ? 2 * BM : BM, NT, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      // arrive on the same barrier of every CTA of the pair once the MMAs issued so far have retired
      auto commit = [&](uint64_t* bar) {
        if (PAIR) {
          umma_commit_pair(mapa_u32(smem_u32(bar), 0));
          umma_commit_pair(mapa_u32(smem_u32(bar), 1));
        } else {
          umma_commit(bar);
        }
      };
      for (long long tile = worker; tile < total_tiles && !*abort_flag; tile += num_workers) {
        const TileCoord t = decode_tile<SCHED, TM>(p, tile, m_tiles, n_tiles);
        if (!mbar_wait(&tmem_empty[acc], acc_phase ^ 1)) {
          *abort_flag = 1;
          atomicExch(p.status, 2);
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (MT == 2 ? 0 : acc * NT);
        bool failed = false;
        for (int kb = 0; kb < t.k_blocks; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase)) {
            failed = true;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t db = B_MN ? umma_smem_desc(sb + k * 2048, 8192, 1024) : umma_smem_desc(sb + k * 32, 16, 1024);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
              const uint32_t sai = sa + i * A_SUB_BYTES;
              const uint64_t da = A_MN ? umma_smem_desc(sai + k * 2048, 8192, 1024) : umma_smem_desc(sai + k * 32, 16, 1024);
              if (PAIR) umma_bf16_ss_pair(d_tmem + i * NT, da, db, idesc, (kb | k) != 0);
              else umma_bf16_ss(d_tmem + i * NT, da, db, idesc, (kb | k) != 0);
            }
          }
          commit(&empty_bar[stage]);   // frees the stage once these MMAs have read it
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (failed) {
          *abort_flag = 1;
          atomicExch(p.status, 3);
          break;
        }
        commit(&tmem_full[acc]);
        if (++acc == NACC) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9; EPI_PUSH: 2..5)
    const int quad = warp & 3;                 // TMEM lane group this warp may read
    const int row_in_tile = quad * 32 + lane;
    const int half = (warp - 2) >> 2;          // which half of the tile's columns (EPI_PUSH: all of them)
    // A thread reads one row of the accumulator.  Loads and stores of global memory straight from that layout put 16
    // bytes per lane at 32 rows into one instruction: half sectors, 32 lines.  Instead each warp passes 32 rows x 32
    // fp32 columns through shared memory (16-byte units, XOR-swizzled by row: conflict-free both ways), after which
    // four lanes hold 32 consecutive columns of a row.  Products with a short reduction are bound by this part; before
    // (four warps, straight stores) and after, us: bf16 store 8192 x 3584 K 1024 55 -> 47, SwiGLU 4096 x 14336 K 4096
    // 756 -> 711 and 4096 x 1536 K 1024 45 -> 34.
    uint4* const staged = reinterpret_cast<uint4*>(smem + STAGES * STAGE_BYTES) + (warp - 2) * 256;
    auto swz = [](int r) { return (r & 1) | ((r & 2) << 1) | ((r & 4) >> 1); };
    constexpr bool ACC = EPI == EPI_ACC_F32 || EPI == EPI_ACC_BF16, F32 = EPI == EPI_ACC_F32 || EPI == EPI_STORE_F32;
    const bool add = ACC && p.beta != 0.f;
    const int q = lane & 3;
    // What the epilogue reads from global memory for 32 columns of the warp's rows.  A tile of 64 columns has one such chunk
    // per warp, which is requested before the wait for the product (1024 x 768 K 512 with rotation 6.2 -> 5.5 us); wider
    // tiles request a chunk as they come to it, the product of the next tile hides it.
    constexpr int OLD = EPI == EPI_ACC_BF16 ? 1 : (EPI == EPI_ROPE || EPI == EPI_SWIGLU_BWD) ? 2 : 0;
    constexpr bool EARLY = NT == 64;
    uint4 old[4][OLD ? OLD : 1];
    auto fetch_old = [&](const TileCoord& t, int sub, int c) {
      const long long col = static_cast<long long>(t.n_tile) * NT + c + q * 8;
      if ((ACC && !add) || col >= p.N) return;
      const long long expert_off = SCHED == SCHED_WGRAD ? t.expert * p.d_expert_stride : 0;
      const long long first = static_cast<long long>(t.m_tile) * TILE_M + (PAIR ? static_cast<int>(cta) : sub) * BM + quad * 32;
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        const long long rr = first + it * 8 + (lane >> 2);
        if (rr >= p.M) continue;
        if (EPI == EPI_ACC_BF16) {
          const bool low = !p.d2 || rr < p.m_split;
          old[it][0] = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(low ? p.d : p.d2) + expert_off +
                                                       (low ? rr : rr - p.m_split) * p.ldd + col);
        } else if (EPI == EPI_ROPE && col < p.rope_cols) {
          // four adjacent pairs (2j, 2j+1) of a head: table entries [position][(col mod 128)/2 + j]
          const size_t tab = static_cast<size_t>(static_cast<int>(rr) % p.rope_seq) * 64 + ((col & 127) >> 1);
          old[it][0] = *reinterpret_cast<const uint4*>(p.rope_cos + tab);
          old[it][OLD - 1] = *reinterpret_cast<const uint4*>(p.rope_sin + tab);
        } else if (EPI == EPI_SWIGLU_BWD) {
          old[it][0] = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.d_gate) + rr * p.N + col);
          old[it][OLD - 1] = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.d_up) + rr * p.N + col);
        }
      }
    };
    int acc = 0;
    uint32_t acc_phase = 0;
    for (long long tile = worker; tile < total_tiles && !*abort_flag; tile += num_workers) {
      const TileCoord t = decode_tile<SCHED, TM>(p, tile, m_tiles, n_tiles);
      if (OLD && EARLY) fetch_old(t, 0, half * (NT / 2));
      if (!mbar_wait(&tmem_full[acc], acc_phase)) {
        *abort_flag = 1;
        atomicExch(p.status, 4);
        break;
      }
      tc_fence_after();
      const bool empty_k = t.k_blocks == 0;   // an expert without rows contributes nothing
#pragma unroll 1
      for (int sub = 0; sub < MT; ++sub) {
      const uint32_t taddr = tmem_base + (MT == 2 ? sub * NT : acc * NT) + (static_cast<uint32_t>(quad * 32) << 16);
      const long long row = static_cast<long long>(t.m_tile) * TILE_M + (PAIR ? static_cast<int>(cta) : sub) * BM + row_in_tile;
      const bool row_ok = row < p.M;
      const long long row0 = row - lane;
      if (EPI == EPI_SWIGLU) {
        // 16 gate and 16 up columns at a time; afterwards two lanes per row, eight features each
        __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(p.d);
        const long long half_n = p.N / 2;
        const long long col0 = static_cast<long long>(t.n_tile) * (NT / 2);
        const int q = lane & 1;
#pragma unroll 1
        for (int c = half * (NT / 4); c < (half + 1) * (NT / 4); c += 16) {
          uint32_t g[16], u[16];
          tmem_ld_32x16(taddr + c, g);
          tmem_ld_32x16(taddr + NT / 2 + c, u);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            staged[lane * 8 + (i ^ swz(lane))] = make_uint4(g[4 * i], g[4 * i + 1], g[4 * i + 2], g[4 * i + 3]);
            staged[lane * 8 + ((4 + i) ^ swz(lane))] = make_uint4(u[4 * i], u[4 * i + 1], u[4 * i + 2], u[4 * i + 3]);
          }
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 2; ++it) {
            const int r = it * 16 + (lane >> 1);
            const uint4 ga = staged[r * 8 + ((2 * q) ^ swz(r))], gb = staged[r * 8 + ((2 * q + 1) ^ swz(r))];
            const uint4 ua = staged[r * 8 + ((4 + 2 * q) ^ swz(r))], ub = staged[r * 8 + ((5 + 2 * q) ^ swz(r))];
            const uint32_t gw[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
            const uint32_t uw[8] = {ua.x, ua.y, ua.z, ua.w, ub.x, ub.y, ub.z, ub.w};
            if (row0 + r < p.M && col0 + c < half_n) {
              uint32_t out[4], og[4], ou[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float g0 = __uint_as_float(gw[2 * i]), g1 = __uint_as_float(gw[2 * i + 1]);
                const float u0 = __uint_as_float(uw[2 * i]), u1 = __uint_as_float(uw[2 * i + 1]);
                out[i] = pack_bf16(g0 / (1.f + __expf(-g0)) * u0, g1 / (1.f + __expf(-g1)) * u1);
                og[i] = pack_bf16(g0, g1);
                ou[i] = pack_bf16(u0, u1);
              }
              const long long off = (row0 + r) * half_n + col0 + c + q * 8;
              *reinterpret_cast<uint4*>(h + off) = make_uint4(out[0], out[1], out[2], out[3]);
              if (p.d_gate) {
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.d_gate) + off) = make_uint4(og[0], og[1], og[2], og[3]);
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.d_up) + off) = make_uint4(ou[0], ou[1], ou[2], ou[3]);
              }
            }
          }
          __syncwarp();
        }
      } else if (EPI == EPI_PUSH) {
        // Rows leave for other GPUs.  A thread owns one row of the accumulator, so storing straight from registers
        // would put 16 bytes per lane at 32 different rows in every store instruction.  Instead each warp stages
        // 128 columns of its 32 rows in shared memory (16-byte units XOR-swizzled by row: conflict-free both ways) and
        // writes them out two rows per instruction, 256 contiguous bytes per row.
        const long long col_base = static_cast<long long>(t.n_tile) * BN;
        uint4* stage = reinterpret_cast<uint4*>(smem + STAGES * STAGE_BYTES) + (warp - 2) * (32 * 16);
        int tag = -1, dest = -1;
        float w = 1.f;
        if (row_ok) {
          tag = p.push_tag[row];
          dest = p.push_src[row];
          if (p.push_w) w = p.push_w[row];
          if (dest < 0 || dest >= p.push_n) tag = -1;          // padding row: nobody waits for it
        }
#pragma unroll 1
        for (int half = 0; half < BN / 128; ++half) {
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t v[32];
            tmem_ld_32x32(taddr + half * 128 + c * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 4; ++i)
              stage[lane * 16 + ((c * 4 + i) ^ (lane & 15))] =
                  make_uint4(pack_bf16(w * __uint_as_float(v[8 * i]), w * __uint_as_float(v[8 * i + 1])),
                             pack_bf16(w * __uint_as_float(v[8 * i + 2]), w * __uint_as_float(v[8 * i + 3])),
                             pack_bf16(w * __uint_as_float(v[8 * i + 4]), w * __uint_as_float(v[8 * i + 5])),
                             pack_bf16(w * __uint_as_float(v[8 * i + 6]), w * __uint_as_float(v[8 * i + 7])));
          }
          __syncwarp();
          const int unit = lane & 15;
          const long long col = col_base + half * 128 + unit * 8;
#pragma unroll 4
          for (int pair = 0; pair < 16; ++pair) {
            const int r = pair * 2 + (lane >> 4);
            const int tag_r = __shfl_sync(0xffffffffu, tag, r);
            const int dest_r = __shfl_sync(0xffffffffu, dest, r);
            if (tag_r >= 0 && col < p.N) {
              const uint4 data = stage[r * 16 + (unit ^ (r & 15))];
              *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.push_dst.ptr[dest_r]) +
                                        static_cast<long long>(tag_r) * p.ldd + col) = data;
            }
          }
          __syncwarp();
        }
      } else {
        const long long col_base = static_cast<long long>(t.n_tile) * NT;
        const long long expert_off = SCHED == SCHED_WGRAD ? t.expert * p.d_expert_stride : 0;
        constexpr bool SCALED = EPI == EPI_ACC_F32 || EPI == EPI_ACC_BF16 || EPI == EPI_STORE_BF16 || EPI == EPI_STORE_F32;
        const float alpha = SCALED && p.alpha ? *p.alpha : 1.f;
        if (NT >= 128 && (EPI == EPI_STORE_BF16 || (EPI == EPI_ACC_BF16 && !add))) {
          // Nothing is added to the product: it is rounded before it is staged, 64 columns of a row in 128 bytes.  In fp32 a
          // tile passes 128 KiB each way, 2048 cycles of the shared memory, which a launch with a short reduction or a
          // single tile shows: us, 6144 x 4096 K 100 26.7 -> 22.2, 1024 x 1024 K 1024 10.7 -> 9.7, 100 x 512 K 512 8.0 ->
          // 7.1 (stored straight from the accumulator's layout: 22.1, 10.2 and 7.2).
          const int q8 = lane & 7;
#pragma unroll 1
          for (int c = half * (NT / 2); c < (half + 1) * (NT / 2); c += 64) {
            if (col_base + c >= p.N) break;
            uint32_t v[2][32];
            if (!empty_k) {
              tmem_ld_32x32(taddr + c, v[0]);
              tmem_ld_32x32(taddr + c + 32, v[1]);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int i = 0; i < 64; ++i) v[i >> 5][i & 31] = 0;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              uint32_t w[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const int e = (i & 3) * 8 + 2 * k;
                w[k] = pack_bf16(__uint_as_float(v[i >> 2][e]) * alpha, __uint_as_float(v[i >> 2][e + 1]) * alpha);
              }
              staged[lane * 8 + (i ^ swz(lane))] = make_uint4(w[0], w[1], w[2], w[3]);
            }
            __syncwarp();
            const long long col = col_base + c + q8 * 8;     // N is a multiple of 32 (checked on the host)
#pragma unroll
            for (int it = 0; it < 8; ++it) {
              const int r = it * 4 + (lane >> 3);
              if (row0 + r >= p.M || col >= p.N) continue;
              const bool low = !ACC || !p.d2 || row0 + r < p.m_split;
              const long long off = expert_off + (low ? row0 + r : row0 + r - p.m_split) * p.ldd + col;
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(low ? p.d : p.d2) + off) = staged[r * 8 + (q8 ^ swz(r))];
            }
            __syncwarp();
          }
        }
        if (F32) {
          // fp32 results leave as 32 x 32 boxes that the memory system writes or adds: a warp stages its rows of 32 columns
          // (16-byte units, XOR-swizzled by row as the tensor map has it) and one lane sends them off.  Each value is added once
          // per launch, so results do not depend on the order of the tiles; the addition is the SM's, subnormals included.
          // Before, the warp read the old values, added and stored (the same bits): twice the traffic through the SM, beside
          // the operands of the next tile.  us, before -> now: 8 experts of 3584 x 1024, 1024 rows each 82.7 -> 72.7, both
          // halves in one launch 140.6 -> 130.6 (470 MB of results alone are 73), 768 x 512 K 1024 15.1 -> 12.6, 6144 x 4096 K
          // 16384 575 -> 558.  Reading the old values a chunk ahead instead, or 16 contiguous bytes per lane, gave nothing.
#pragma unroll 1
          for (int c = half * (NT / 2); c < (half + 1) * (NT / 2); c += 32) {
            if (col_base + c >= p.N || row0 >= p.M || (add && empty_k)) break;
            uint32_t v[32];
            if (!empty_k) {
              tmem_ld_32x32(taddr + c, v);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = 0;
            }
            if (ACC && p.d2 && row0 < p.m_split && row0 + 32 > p.m_split) {
              // rows of both results in one warp (a cut that is no multiple of 32): each lane its own row
              if (row_ok) {
                float* dst = reinterpret_cast<float*>(row < p.m_split ? p.d : p.d2) + expert_off +
                             (row < p.m_split ? row : row - p.m_split) * p.ldd + col_base + c;
#pragma unroll
                for (int i = 0; i < 32; ++i) dst[i] = (add ? dst[i] : 0.f) + __uint_as_float(v[i]) * alpha;
              }
              continue;
            }
            if (lane == 0) bulk_wait_read();      // the previous box has left the staging buffer
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i)
              staged[lane * 8 + (i ^ (lane & 7))] = make_uint4(
                  __float_as_uint(__uint_as_float(v[4 * i]) * alpha), __float_as_uint(__uint_as_float(v[4 * i + 1]) * alpha),
                  __float_as_uint(__uint_as_float(v[4 * i + 2]) * alpha), __float_as_uint(__uint_as_float(v[4 * i + 3]) * alpha));
            fence_async_shared();
            __syncwarp();
            if (lane == 0) {
              const int col = static_cast<int>(col_base) + c, r = static_cast<int>(row0);
              const bool low = !ACC || !p.d2 || r < p.m_split;
              const CUtensorMap* map = low ? &p.map_d : &p.map_d2;
              const int expert = SCHED == SCHED_WGRAD ? t.expert : 0;
              if (add) tma_add_3d(map, staged, col, low ? r : r - p.m_split, expert);
              else tma_store_3d(map, staged, col, low ? r : r - p.m_split, expert);
              bulk_commit();
            }
          }
        }
#pragma unroll 1
        for (int c = half * (NT / 2);
             !F32 && (NT < 128 || (EPI != EPI_STORE_BF16 && (EPI != EPI_ACC_BF16 || add))) && c < (half + 1) * (NT / 2); c += 32) {
          const long long col = col_base + c + q * 8;     // N is a multiple of 32 (checked on the host)
          if (col_base + c >= p.N) break;
          if (OLD && !EARLY) fetch_old(t, sub, c);
          uint32_t v[32];
          if (!empty_k) {
            tmem_ld_32x32(taddr + c, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
            staged[lane * 8 + (i ^ swz(lane))] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int r = it * 8 + (lane >> 2);
            const uint4 a = staged[r * 8 + ((2 * q) ^ swz(r))], b = staged[r * 8 + ((2 * q + 1) ^ swz(r))];
            float x[8] = {__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(a.w),
                          __uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z), __uint_as_float(b.w)};
            const uint4 o0 = old[it][0], o1 = old[it][OLD ? OLD - 1 : 0];
            const uint32_t w0[4] = {o0.x, o0.y, o0.z, o0.w}, w1[4] = {o1.x, o1.y, o1.z, o1.w};
            if (row0 + r >= p.M) continue;
            if (SCALED) {
#pragma unroll
              for (int i = 0; i < 8; ++i) x[i] = __fmul_rn(x[i], alpha);     // rounded before the addition on every tile kind
            }
            const bool low = !ACC || !p.d2 || row0 + r < p.m_split;
            const long long off = expert_off + (low ? row0 + r : row0 + r - p.m_split) * p.ldd + col;
            void* const out = low ? p.d : p.d2;
            if (EPI == EPI_SWIGLU_BWD) {
              uint32_t og[4], ou[4], oh[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w0[j]));
                const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w1[j]));
                const float s0 = 1.f / (1.f + __expf(-g.x)), s1 = 1.f / (1.f + __expf(-g.y));
                const float l0 = g.x * s0, l1 = g.y * s1;
                og[j] = pack_bf16(x[2 * j] * u.x * s0 * (1.f + g.x * (1.f - s0)),
                                  x[2 * j + 1] * u.y * s1 * (1.f + g.y * (1.f - s1)));
                ou[j] = pack_bf16(x[2 * j] * l0, x[2 * j + 1] * l1);
                oh[j] = pack_bf16(l0 * u.x, l1 * u.y);
              }
              __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.d) + off;
              *reinterpret_cast<uint4*>(dst) = make_uint4(og[0], og[1], og[2], og[3]);
              *reinterpret_cast<uint4*>(dst + p.N) = make_uint4(ou[0], ou[1], ou[2], ou[3]);
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.h) + (row0 + r) * p.N + col) =
                  make_uint4(oh[0], oh[1], oh[2], oh[3]);
            } else {
              if (EPI == EPI_ACC_BF16 && add) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 prev = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w0[j]));
                  x[2 * j] = __fadd_rn(x[2 * j], prev.x);
                  x[2 * j + 1] = __fadd_rn(x[2 * j + 1], prev.y);
                }
              }
              if (EPI == EPI_ROPE && col < p.rope_cols) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float cv = __uint_as_float(w0[j]), sv = __uint_as_float(w1[j]);
                  const float x0 = x[2 * j], x1 = x[2 * j + 1];
                  x[2 * j] = x0 * cv - x1 * sv;
                  x[2 * j + 1] = x0 * sv + x1 * cv;
                }
              }
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(out) + off) =
                  make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
            }
          }
          __syncwarp();
        }
      }
      }  // sub
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty[acc]), 0));
        else mbar_arrive(&tmem_empty[acc]);
      }
      if (++acc == NACC) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if ((EPI == EPI_ACC_F32 || EPI == EPI_STORE_F32) && lane == 0) bulk_wait();      // this warp's stores are done
  }

  if (EPI == EPI_PUSH) __threadfence_system();   // my rows are in the peers' memory before the flag below
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();   // the peer's shared memory, barriers and tensor memory are idle as well
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
  if (EPI == EPI_PUSH && threadIdx.x == 0) {
    // the last CTA to get here tells every rank that this rank's rows have been delivered
    const unsigned int old = atomicInc(p.push_ticket, gridDim.x - 1);
    if (old == gridDim.x - 1) {
      __threadfence_system();
      signal_all(p.push_sig, p.push_slot, p.push_rank, p.push_n, p.push_seq);
    }
  }
}

// ------------------------------------------------------------------ host side
template <int A_MN, int B_MN, int EPI, int SCHED, int MT, int NT = BN>
static int launch_mt(const GemmParams& p, int sms, cudaStream_t stream) {
  auto kernel = gemm_tcgen05_kernel<A_MN, B_MN, EPI, SCHED, MT, 0, NT>;
  constexpr int smem = smem_bytes<EPI, MT, 0, NT>();
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -3;
    configured = true;
  }
  const long long tiles = static_cast<long long>((p.M + MT * BM - 1) / (MT * BM)) * ((p.N + NT - 1) / NT) *
                          (SCHED == SCHED_WGRAD ? p.num_experts : 1);
  // a CTA per tile where that is less than one per SM (the return of an expert group counts its CTAs: always all)
  const int grid = EPI != EPI_PUSH && tiles < sms ? static_cast<int>(tiles < 1 ? 1 : tiles) : sms;
  if (EPI == EPI_PUSH) kernel<<<grid, gemm_threads<EPI>(), smem, stream>>>(p);
  else launch_next(kernel, grid, gemm_threads<EPI>(), smem, stream, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// CTA pairs: a cluster of two CTAs per 256x256 tile, as many pairs as the device keeps resident.
// Returns -20 when clusters of two with this much shared memory cannot be scheduled.
template <int A_MN, int B_MN, int EPI, int SCHED>
static int pairs_resident(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int sms) {
  auto kernel = gemm_tcgen05_kernel<A_MN, B_MN, EPI, SCHED, 1, 1>;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg->blockDim = dim3(gemm_threads<EPI>());
  cfg->dynamicSmemBytes = smem_bytes<EPI, 1, 1>();
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  static int max_pairs = -1;
  if (max_pairs < 0) {
    max_pairs = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<EPI, 1, 1>()) == cudaSuccess) {
      int clusters = 0;
      cfg->gridDim = dim3(sms / 2 * 2);
      if (cudaOccupancyMaxActiveClusters(&clusters, kernel, cfg) == cudaSuccess) max_pairs = clusters;
      else cudaGetLastError();
    }
  }
  return max_pairs;
}

template <int A_MN, int B_MN, int EPI, int SCHED>
static int launch_pair(const GemmParams& p, int sms, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  const int pairs = pairs_resident<A_MN, B_MN, EPI, SCHED>(&cfg, attr, sms);
  if (pairs < 1) return -20;
  cfg.gridDim = dim3(2 * pairs);
  cfg.stream = stream;
  cfg.numAttrs = EPI == EPI_PUSH ? 1 : 2;      // chain.cuh
  if (cudaLaunchKernelEx(&cfg, gemm_tcgen05_kernel<A_MN, B_MN, EPI, SCHED, 1, 1>, p) != cudaSuccess) {
    cudaGetLastError();
    return -4;
  }
  return 0;
}

static int g_tile_mode = 0;   // 0 auto, 1 force 128x256, 2 force 256x256 on one CTA, 3 force CTA pairs where legal, 4 auto
                              // (EPI_PUSH included), 5 auto among the single-CTA kinds

enum TileKind : int { TILE_128 = 0, TILE_256 = 1, TILE_PAIR = 2, TILE_N128 = 3, TILE_N64 = 4 };

// Rows of one box of a K-major B operand (SwiGLU: of each of its two weights).
static int box_rows(TileKind kind, bool swiglu = false) {
  if (swiglu) return kind == TILE_N64 ? 32 : kind == TILE_N128 ? 64 : 128;
  return kind == TILE_N64 ? 64 : kind == TILE_N128 || kind == TILE_PAIR ? 128 : 256;
}

// 256-row tiles (one CTA with two sub-tiles, or a CTA pair) need whole 256-row tiles of one expert: the caller says
// whether its segments are padded to 256 rows.
// 256x256 on one CTA for long reductions over many tiles: the exposed epilogue is amortised, and it takes the least energy
// per operation (down projection of 11 000 expert rows, K 14336: 0.96 ms against 1.02-1.10 ms on pairs; its dx, K 28672:
// 1.82 against 1.96-2.15).  Otherwise CTA pairs wherever their tiles reach half of the machine's pairs.  Whole passes,
// single-CTA kinds only -> this rule: three-layer dense SwiGLU stack 11.28 -> 10.36 ms, one-block step of 2 x 16384 tokens
// 107.5 -> 103.0, head and loss of 6001 tokens 2.17 -> 2.07.  The eight-block step that runs against the 1000 W power cap
// for ten seconds, ms: single-CTA kinds only 10510, pairs for everything large 10540, this rule 10237.  Below that 128x256
// on one CTA.  The expert-parallel return (EPI_PUSH) stays with the single-CTA kinds: its time depends on the links, which
// one GPU does not show.
template <int SCHED, int EPI>
static TileKind choose_tile(const GemmParams& p, int sms, bool pair_available) {
  const long long k_eff = SCHED == SCHED_WGRAD ? p.K / (p.num_experts > 0 ? p.num_experts : 1) : p.K;
  const bool legal = SCHED == SCHED_WGRAD ||
                     (p.tile_expert == nullptr ? p.num_m_tiles == nullptr : p.group_align256 != 0);
  const long long columns = static_cast<long long>((p.N + BN - 1) / BN) * (SCHED == SCHED_WGRAD ? p.num_experts : 1);
  const long long tiles256 = (p.M + 255) / 256 * columns, tiles128 = (p.M + 127) / 128 * columns;
  if (EPI != EPI_PUSH && (g_tile_mode == 6 || g_tile_mode == 7)) return g_tile_mode == 6 ? TILE_N128 : TILE_N64;
  if (EPI != EPI_PUSH && (g_tile_mode == 0 || g_tile_mode == 4 || g_tile_mode == 5)) {
    // Narrow tiles.  A step of 64 along k takes a CTA 0.27 us at 256 columns and 0.16 at 128 or 64 (its loads bound it), so
    // tiles of 128 columns win where their waves are fewer than 1.6 times those of 256: one wave instead of one, up to three
    // instead of two.  64 columns take as long as 128 along k and half as long in the epilogue: where they make one wave.
    // Grouped rows: an expert's padding to 256 rows is half of that on average.  us, 256 -> 128 -> 64 columns: 1024 x 512 K
    // 512 7.3, 5.6, 5.3; 2048 x 1024 K 1024 10.0, 7.4, 9.6 (two waves); 4096 x 1536 K 1024 16.3, 14.8, 20.7; fp32 gradient
    // 768 x 512 K 1024 12.4, 8.4, 6.9, 1024 x 1024 K 4096 25.7, 16.3, 14.6; but 4096 x 1024 K 1024 10.4, 11.1, 15.0.
    const long long rows = p.num_m_tiles ? max(128, p.M - 128 * p.num_experts) : p.M;
    const long long groups = SCHED == SCHED_WGRAD ? p.num_experts : 1;
    const auto waves = [&](int width) { return ((rows + 127) / 128 * ((p.N + width - 1) / width) * groups + sms - 1) / sms; };
    const long long w256 = waves(256), w128 = waves(128);
    if (waves(64) == 1) {
      // Loads of an A operand below 128 KiB are slow, whatever its shape (4096 columns, 64 CTAs: K 4096 21.4 us at 15 rows and 12.9
      // at 16, K 8192 37.8 at 6 and 22.4 at 8), and the slower the more CTAs read it: 128 columns where 64 make more than 32 CTAs
      // (6144 columns, one row, K 4096: 64 columns 28, 128 21.9, 256 22; 4096 columns 21.4, 16.4, 21.9).
      const bool small_a = SCHED == SCHED_FLAT && static_cast<long long>(p.M) * p.K * 2 < 128 * 1024;
      return small_a && (p.N + 63) / 64 > 32 ? TILE_N128 : TILE_N64;
    }
    if (w128 == 1 || (w256 == 2 && w128 == 3)) return TILE_N128;
  }
  if (!legal || g_tile_mode == 1) return TILE_128;
  if (g_tile_mode == 2) return TILE_256;
  if (pair_available && g_tile_mode == 3) return TILE_PAIR;
  if (g_tile_mode == 3) return TILE_128;
  const bool pairs = g_tile_mode == 4 || (g_tile_mode == 0 && EPI != EPI_PUSH);
  if (tiles256 >= 2LL * sms && k_eff >= 6144) return TILE_256;
  // Where the second half of the last row of pair tiles lies behind the matrix, pairs may need a wave more: not where it
  // is more than the tenth that they gain per wave.  Loss of one token, 32000 entries, width 4096: 75 us on 125 pair
  // tiles (two waves of 74), 61 on 125 single ones (one of 148); 100 tokens, width 512: 22.8 and 16.0.
  const long long waves256 = (tiles256 + sms / 2 - 1) / (sms / 2), waves128 = (tiles128 + sms - 1) / sms;
  return pair_available && pairs && tiles256 >= sms / 2 && 10 * waves256 <= 11 * waves128 ? TILE_PAIR : TILE_128;
}

template <int A_MN, int B_MN, int EPI, int SCHED>
static bool pair_available(int sms) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  return pairs_resident<A_MN, B_MN, EPI, SCHED>(&cfg, attr, sms) >= sms / 2 - 8;   // (nearly) every SM in a pair
}

template <int A_MN, int B_MN, int EPI, int SCHED>
static int launch(const GemmParams& p, TileKind kind, int sms, cudaStream_t stream) {
  if constexpr (EPI != EPI_PUSH) {
    if (kind == TILE_N128) return launch_mt<A_MN, B_MN, EPI, SCHED, 1, 128>(p, sms, stream);
    if (kind == TILE_N64) return launch_mt<A_MN, B_MN, EPI, SCHED, 1, 64>(p, sms, stream);
  }
  if (kind == TILE_PAIR) return launch_pair<A_MN, B_MN, EPI, SCHED>(p, sms, stream);
  if (kind == TILE_256) return launch_mt<A_MN, B_MN, EPI, SCHED, 2>(p, sms, stream);
  return launch_mt<A_MN, B_MN, EPI, SCHED, 1>(p, sms, stream);
}

// Convenience for entry points whose tensor maps do not depend on the tile kind.
template <int A_MN, int B_MN, int EPI, int SCHED>
static int launch(const GemmParams& p, int sms, cudaStream_t stream) {
  return launch<A_MN, B_MN, EPI, SCHED>(p, choose_tile<SCHED, EPI>(p, sms, pair_available<A_MN, B_MN, EPI, SCHED>(sms)),
                                        sms, stream);
}

static int sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return sms;
}

}  // namespace b2

using namespace b2;

// Arguments shared by the entry points below:
//   a, b           bf16 operands; layouts per entry point
//   lda, ldb       row pitch in elements
//   tile_expert    optional int32 [ceil(M/128)] expert of each 128-row tile (grouped problems)
//   num_m_tiles    optional device int32 scalar with the live tile count
//   status         device int32 word, set non-zero if an in-kernel wait ran out
extern "C" {

// 0 automatic, 1 always 128x256 tiles, 2 single-CTA 256x256 tiles wherever they are legal, 3 CTA pairs wherever legal,
// 4 automatic for the expert-parallel return too, 5 automatic among the single-CTA kinds, 6 and 7 tiles of 128 and of 64
// columns.
void b2_gemm_set_tile_mode(int mode) { g_tile_mode = mode; }

// y[M,N] = a[M,K] * w[e][N,K]^T      (a K-major, w K-major)
// epi: 0 bf16 store, 4 fp32 store.
int b2_gemm_nt(const void* a, const void* w, void* d, int M, int N, int K, long long lda, long long ldw,
               long long ldd, int num_experts, const int* tile_expert, const int* num_m_tiles, int group_align256,
               int epi, int* status, cudaStream_t stream) {
  if (N % 32 || K % 8) return -10;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.num_experts = num_experts; p.b_expert_rows = N; p.k_split = 0;
  p.tile_expert = tile_expert; p.num_m_tiles = num_m_tiles; p.d = d; p.ldd = ldd; p.status = status; p.beta = 0.f;
  p.group_align256 = group_align256;
  if (epi != EPI_STORE_BF16 && epi != EPI_STORE_F32) return -13;
  const int sms = sm_count();
  const bool pairs = epi == EPI_STORE_BF16 ? pair_available<0, 0, EPI_STORE_BF16, SCHED_FLAT>(sms)
                                           : pair_available<0, 0, EPI_STORE_F32, SCHED_FLAT>(sms);
  const TileKind kind = choose_tile<SCHED_FLAT, EPI_STORE_BF16>(p, sms, pairs);
  if (make_map(&p.map_a, a, K, M, lda, BM)) return -11;
  // a CTA of a pair stages 128 of the tile's 256 weight rows
  if (make_map(&p.map_b, w, K, static_cast<long long>(num_experts) * N, ldw, box_rows(kind))) return -12;
  if (epi == EPI_STORE_BF16) return launch<0, 0, EPI_STORE_BF16, SCHED_FLAT>(p, kind, sms, stream);
  if (make_out_map(&p.map_d, d, N, M, 1, ldd, M * ldd)) return -14;
  return launch<0, 0, EPI_STORE_F32, SCHED_FLAT>(p, kind, sms, stream);
}

// h[M,F] = silu(a w1[e]^T) * (a w3[e]^T); optional gate/up pre-activations [M,F].
int b2_gemm_swiglu(const void* a, const void* w1, const void* w3, void* h, void* gate, void* up, int M, int F, int K,
                   long long lda, int num_experts, const int* tile_expert, const int* num_m_tiles, int group_align256,
                   int* status, cudaStream_t stream) {
  if (F % 128 || K % 8) return -10;
  GemmParams p{};
  p.M = M; p.N = 2 * F; p.K = K; p.num_experts = num_experts; p.b_expert_rows = F; p.k_split = 0;
  p.tile_expert = tile_expert; p.num_m_tiles = num_m_tiles; p.d = h; p.d_gate = gate; p.d_up = up; p.ldd = F;
  p.status = status; p.group_align256 = group_align256;
  const int sms = sm_count();
  const TileKind kind = choose_tile<SCHED_FLAT, EPI_SWIGLU>(p, sms, pair_available<0, 0, EPI_SWIGLU, SCHED_FLAT>(sms));
  if (make_map(&p.map_a, a, K, M, lda, BM)) return -11;
  if (make_map(&p.map_b, w1, K, static_cast<long long>(num_experts) * F, K, box_rows(kind, true))) return -12;
  if (make_map(&p.map_b2, w3, K, static_cast<long long>(num_experts) * F, K, box_rows(kind, true))) return -12;
  return launch<0, 0, EPI_SWIGLU, SCHED_FLAT>(p, kind, sms, stream);
}

// dx[M,N] = a[M,K] * w[e][K,N]     (w MN-major: its rows are the reduction index).
// ``alpha`` (optional device scalar) multiplies the result.
// If w2 is given, K = k_split + K2 and rows k >= k_split come from w2 (dx = dg W1 + du W3 in one pass).
int b2_gemm_nn(const void* a, const void* w, const void* w2, void* d, int M, int N, int K, int k_split, long long lda,
               long long ldw, long long ldd, int num_experts, const int* tile_expert, const int* num_m_tiles,
               int group_align256, const float* alpha, int* status, cudaStream_t stream) {
  if (N % 32 || K % 64 || (w2 && k_split % 64)) return -10;
  GemmParams p{};
  p.alpha = alpha;
  const int rows = w2 ? k_split : K;
  if (make_map(&p.map_a, a, K, M, lda, BM)) return -11;
  if (make_map(&p.map_b, w, N, static_cast<long long>(num_experts) * rows, ldw, 64)) return -12;
  if (w2 && make_map(&p.map_b2, w2, N, static_cast<long long>(num_experts) * (K - k_split), ldw, 64)) return -12;
  p.M = M; p.N = N; p.K = K; p.num_experts = num_experts; p.b_expert_rows = rows; p.k_split = w2 ? k_split : 0;
  p.tile_expert = tile_expert; p.num_m_tiles = num_m_tiles; p.d = d; p.ldd = ldd; p.status = status;
  p.group_align256 = group_align256;
  return launch<0, 1, EPI_STORE_BF16, SCHED_FLAT>(p, sm_count(), stream);
}

// SwiGLU backward of the hidden layer in one launch: dh[M,F] = a[M,K] * w[e][K,F] stays in tensor memory; with the saved
// pre-activations gate, up [M,F] the epilogue stores dgu[M,2F] = [dh u silu'(g) | dh silu(g)] and h[M,F] = silu(g) u.
int b2_gemm_nn_swiglu_bwd(const void* a, const void* w, const void* gate, const void* up, void* dgu, void* h, int M,
                          int F, int K, long long lda, int num_experts, const int* tile_expert, const int* num_m_tiles,
                          int group_align256, int* status, cudaStream_t stream) {
  if (F % 32 || K % 64) return -10;
  GemmParams p{};
  if (make_map(&p.map_a, a, K, M, lda, BM)) return -11;
  if (make_map(&p.map_b, w, F, static_cast<long long>(num_experts) * K, F, 64)) return -12;
  p.M = M; p.N = F; p.K = K; p.num_experts = num_experts; p.b_expert_rows = K;
  p.tile_expert = tile_expert; p.num_m_tiles = num_m_tiles; p.group_align256 = group_align256;
  p.d = dgu; p.ldd = 2LL * F; p.h = h; p.d_gate = const_cast<void*>(gate); p.d_up = const_cast<void*>(up);
  p.status = status;
  return launch<0, 1, EPI_SWIGLU_BWD, SCHED_FLAT>(p, sm_count(), stream);
}

// y[M,N] = a[M,K] * w[N,K]^T with the rotary embedding applied to columns [0, rope_cols) in the epilogue: column c
// belongs to head c / 128, pairs (2j, 2j+1) inside a head are rotated by the angle of table entry
// [row mod seq][j] (cos, sin: fp32 [seq, 64]).  rope_cols is a multiple of 128.
int b2_gemm_nt_rope(const void* a, const void* w, void* d, int M, int N, int K, long long lda, long long ldd,
                    const float* cos_t, const float* sin_t, int rope_cols, int seq, int* status,
                    cudaStream_t stream) {
  if (N % 32 || K % 8 || rope_cols % 128 || rope_cols > N || seq < 1) return -10;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.num_experts = 1; p.b_expert_rows = N; p.k_split = 0;
  p.d = d; p.ldd = ldd; p.status = status; p.beta = 0.f;
  p.rope_cos = cos_t; p.rope_sin = sin_t; p.rope_cols = rope_cols; p.rope_seq = seq;
  const int sms = sm_count();
  const TileKind kind = choose_tile<SCHED_FLAT, EPI_ROPE>(p, sms, pair_available<0, 0, EPI_ROPE, SCHED_FLAT>(sms));
  if (make_map(&p.map_a, a, K, M, lda, BM)) return -11;
  if (make_map(&p.map_b, w, K, N, K, box_rows(kind))) return -12;
  return launch<0, 0, EPI_ROPE, SCHED_FLAT>(p, kind, sms, stream);
}

static void fill_push(GemmParams& p, const unsigned long long* dst, const int* tag, const int* src, const float* w,
                      const unsigned long long* sig, int slot, int seq, int rank, int n, unsigned int* ticket) {
  for (int i = 0; i < MAX_RANKS; ++i) {
    p.push_dst.ptr[i] = i < n ? reinterpret_cast<void*>(dst[i]) : nullptr;
    p.push_sig.ptr[i] = i < n ? reinterpret_cast<void*>(sig[i]) : nullptr;
  }
  p.push_tag = tag; p.push_src = src; p.push_w = w; p.push_slot = slot; p.push_seq = seq; p.push_rank = rank;
  p.push_n = n; p.push_ticket = ticket;
}

// Expert-parallel return fused into the epilogue.  The product a[M,K] * w[e][N,K]^T (NT) is not stored locally: row r
// is scaled by push_w[r] (null: 1) and written as bf16 into row push_tag[r] of rank push_src[r]'s buffer
// (``push_dst``: MAX_RANKS device addresses, row pitch N); rows with a negative tag are skipped.  When all CTAs are
// done the kernel writes ``seq`` into slot ``sig_slot`` of every rank's signal pad.  ``ticket``: a zero-initialised
// device word that the kernel leaves at zero.
int b2_gemm_nt_push(const void* a, const void* w, int M, int N, int K, long long lda, int num_experts,
                    const int* tile_expert, const int* num_m_tiles, int group_align256,
                    const unsigned long long* push_dst, const int* push_tag, const int* push_src, const float* push_w,
                    const unsigned long long* sig, int sig_slot, int seq, int rank, int n, unsigned int* ticket,
                    int* status, cudaStream_t stream) {
  if (N % 32 || K % 8 || n < 1 || n > MAX_RANKS) return -10;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.num_experts = num_experts; p.b_expert_rows = N; p.k_split = 0;
  p.tile_expert = tile_expert; p.num_m_tiles = num_m_tiles; p.d = nullptr; p.ldd = N; p.status = status;
  p.group_align256 = group_align256;
  fill_push(p, push_dst, push_tag, push_src, push_w, sig, sig_slot, seq, rank, n, ticket);
  const int sms = sm_count();
  const TileKind kind = choose_tile<SCHED_FLAT, EPI_PUSH>(p, sms, pair_available<0, 0, EPI_PUSH, SCHED_FLAT>(sms));
  if (make_map(&p.map_a, a, K, M, lda, BM)) return -11;
  if (make_map(&p.map_b, w, K, static_cast<long long>(num_experts) * N, K, box_rows(kind)))
    return -12;
  return launch<0, 0, EPI_PUSH, SCHED_FLAT>(p, kind, sms, stream);
}

// The same for a[M,K] * w[e][K,N] with the reduction continued over w2 (dx = dgate W1 + dup W3).
int b2_gemm_nn_push(const void* a, const void* w, const void* w2, int M, int N, int K, int k_split, long long lda,
                    int num_experts, const int* tile_expert, const int* num_m_tiles, int group_align256,
                    const unsigned long long* push_dst, const int* push_tag, const int* push_src, const float* push_w,
                    const unsigned long long* sig, int sig_slot, int seq, int rank, int n, unsigned int* ticket,
                    int* status, cudaStream_t stream) {
  if (N % 32 || K % 64 || (w2 && k_split % 64) || n < 1 || n > MAX_RANKS) return -10;
  GemmParams p{};
  const int rows = w2 ? k_split : K;
  if (make_map(&p.map_a, a, K, M, lda, BM)) return -11;
  if (make_map(&p.map_b, w, N, static_cast<long long>(num_experts) * rows, N, 64)) return -12;
  if (w2 && make_map(&p.map_b2, w2, N, static_cast<long long>(num_experts) * (K - k_split), N, 64)) return -12;
  p.M = M; p.N = N; p.K = K; p.num_experts = num_experts; p.b_expert_rows = rows; p.k_split = w2 ? k_split : 0;
  p.tile_expert = tile_expert; p.num_m_tiles = num_m_tiles; p.d = nullptr; p.ldd = N; p.status = status;
  p.group_align256 = group_align256;
  fill_push(p, push_dst, push_tag, push_src, push_w, sig, sig_slot, seq, rank, n, ticket);
  return launch<0, 1, EPI_PUSH, SCHED_FLAT>(p, sm_count(), stream);
}

// dw[e][M,N] (+)= a[rows_e, M]^T * b[rows_e, N]   (both MN-major; rows_e from cumulative offsets, or all R rows
// when expert_offsets is null).  out_kind: 1 fp32 (+= if beta), 2 bf16 (+= if beta).  ``alpha`` (optional device scalar)
// multiplies the product before it is added.
// With d2 the rows [m_split, M) of the product go to d2 (two weight gradients that share b, in one launch).
// ``expert_counts`` (optional): rows of each segment that count; the rest of the segment holds zeros.
int b2_gemm_tn(const void* a, const void* b, void* d, void* d2, int m_split, int M, int N, int R, long long lda,
               long long ldb, long long ldd, int num_experts, const int* expert_offsets, const int* expert_counts,
               int out_kind, float beta, const float* alpha, int* status, cudaStream_t stream) {
  if (N % 32 || M % 8 || (d2 && (m_split < 1 || m_split >= M))) return -10;
  GemmParams p{};
  p.d2 = d2;
  p.m_split = m_split;
  p.expert_counts = expert_counts;
  p.alpha = alpha;
  if (make_map(&p.map_a, a, M, R, lda, 64)) return -11;
  if (make_map(&p.map_b, b, N, R, ldb, 64)) return -12;
  p.M = M; p.N = N; p.K = R; p.num_experts = num_experts; p.b_expert_rows = 0; p.k_split = 0;
  p.expert_offsets = expert_offsets; p.d = d; p.ldd = ldd; p.d_expert_stride = static_cast<long long>(d2 ? m_split : M) * ldd;
  p.beta = beta; p.status = status;
  if (out_kind == 1) {
    const long long low = d2 ? m_split : M;
    if (make_out_map(&p.map_d, d, N, low, num_experts, ldd, low * ldd)) return -14;
    if (d2 && make_out_map(&p.map_d2, d2, N, M - m_split, num_experts, ldd, low * ldd)) return -14;
  }
  if (expert_offsets) {
    if (out_kind == 1) return launch<1, 1, EPI_ACC_F32, SCHED_WGRAD>(p, sm_count(), stream);
    if (out_kind == 2) return launch<1, 1, EPI_ACC_BF16, SCHED_WGRAD>(p, sm_count(), stream);
  } else {
    if (out_kind == 1) return launch<1, 1, EPI_ACC_F32, SCHED_FLAT>(p, sm_count(), stream);
    if (out_kind == 2) return launch<1, 1, EPI_ACC_BF16, SCHED_FLAT>(p, sm_count(), stream);
  }
  return -13;
}

}  // extern "C"
