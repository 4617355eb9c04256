// Grouped 2:4-sparse int4 delta GEMM for prefill-sized token tiles on the SPARSE fifth-generation
// tensor-core instruction: tcgen05.mma.sp (kind::f16, K = 32 dense per instruction), A operand = the
// STORED halves of the 2:4 weights and their 2:4 metadata, both in tensor memory, B operand = the
// activation tile in shared memory, fp32 accumulator in tensor memory.
//
// Two CTAs of a cluster issue one tcgen05.mma.sp.cta_group::2 per instruction: M = 256 output features
// (128 per CTA: each CTA decodes its own stripe and holds its own accumulator, weights and metadata) x
// N = 64, 128 or 256 tokens, the smallest that holds the tile (each CTA stages half of them).  The
// leader CTA's MMA thread issues for both; every decode warp of both CTAs arrives on the leader's
// barrier; tcgen05.commit with a CTA mask hands stages back to both.
//
// Per 128-K chunk (one scale group, four instructions) and per CTA:
//   producer warps  TMA, one thread each: the activation tile [tokens x 128 K] as two 128-byte-swizzled
//                   halves in one 3-D box (the B operand as it lands) / packed weights, metadata and
//                   scales of the CTA's 128 columns
//   12 decode warps three teams of four (one warp per TMEM lane quadrant) on alternate chunks; a lane owns
//                   one feature: its nibbles -> fp16 (x group scale) -> tcgen05.st into the A columns of
//                   the stage, 8 columns per 32-K slab, and its metadata cells.  The packed format already
//                   holds, per slab, one 16-bit field per row and K half in the tensor core's ordered
//                   2-bit-index form, so a metadata cell (lane = 16*(row/16) + 8*(K half) + row%8) is two
//                   such fields (rows r and r + 8) picked from two packed words with one PRMT
//   MMA warp        one thread issues 4 tcgen05.mma.sp per chunk; a slab's metadata is one column of a
//                   pair, the instruction descriptor's id2 selects it; tcgen05.commit hands the stage back
//   8 epilogue warps tcgen05.ld, scale, convert, transpose 32 x 32 blocks through shared memory and
//                   store 16-byte pieces (8 features of one token)
// TMEM: columns [0, 256) accumulator (one of 256 tokens, or two of up to 128 in turn, so that the
// epilogue of a small tile overlaps the next one's chunks), then 32 columns of weights and 4 of metadata
// per stage.
//
// What bounds it (in-kernel cycle counters): a loop of latencies over the five stages, load about 1200 to 1500
// cycles, decode 700, MMA and hand-back 500: a fifth of that, 480 to 540 cycles, is the least a chunk of 128 K takes.
// Measured 520 (narrow tiles) to 650 (256 tokens), where the instruction itself takes 494 at 256 tokens; and for
// 256-token tiles the drain of the accumulator, about 4000 cycles an item.  The shared-memory
// pipe would be next: 512 wavefronts of activations landing and read, 50 of packed weights, about 100 of decode;
// weights in shared memory would add 256 and a proxy fence on the decode warps' chain.
// Measured, whole calls (before: weights through shared memory, 64-K stages, every tile as 256 tokens, one
// accumulator): 8192 tokens in 16 segments, 5120 -> 13824: 858 -> 705 us; 1531 tokens, one weight, 4096 -> 11008:
// 109 -> 89 us; 700 tokens over 13 deltas (54 each), 4096 -> 12288: 228 -> 116 us.
// Every wait is bounded; both CTAs of a pair meet at a cluster barrier before either leaves.
#pragma once

#include "tc_common.cuh"

namespace trb {

struct TcSpCfg {
  static constexpr int CTAS = 2;            // CTAs of a cluster that share a work item
  static constexpr int TT = 256;            // largest token tile
  static constexpr int SW = 4;              // 64-column blocks per work item (128 columns per CTA)
  static constexpr int KC = 128;            // dense K per stage: one scale group, four sparse MMAs
  static constexpr int SLABS = KC / 32;
  static constexpr int STAGES = 5;
  static constexpr int TEAMS = 3;           // teams of 4 decode warps take alternate chunks
  static constexpr int DECODE0 = 4;         // warps 0-2: activation TMA, MMA, weight TMA; 3 idle (quadrants start at a multiple of 4)
  static constexpr int EPI0 = DECODE0 + 4 * TEAMS;
  static constexpr int EPI_WARPS = 8;       // two per TMEM lane quadrant
  static constexpr int THREADS = (EPI0 + EPI_WARPS) * 32;
  static constexpr int B_BYTES = (TT / CTAS) * KC * 2;   // 32 KiB per CTA at 256 tokens
  static constexpr int Q_BYTES = SLABS * 256 * 4;
  static constexpr int M_BYTES = SLABS * 128 * 4;
  static constexpr int S_BYTES = 256;
  static constexpr int B_OFF = 0;
  static constexpr int Q_OFF = B_OFF + B_BYTES;
  static constexpr int M_OFF = Q_OFF + Q_BYTES;
  static constexpr int S_OFF = M_OFF + M_BYTES;
  static constexpr int STAGE_BYTES = (S_OFF + S_BYTES + 1023) / 1024 * 1024;
  static constexpr int ROWS_OFF = STAGES * STAGE_BYTES;                   // int [TT] output rows
  static constexpr int XPOSE_OFF = ROWS_OFF + TT * 4;                     // [EPI_WARPS][32 tokens][32 features] halves
  static constexpr int PREFIX_OFF = XPOSE_OFF + EPI_WARPS * 2048;
  static constexpr int BAR_OFF = PREFIX_OFF + (kMaxSegments + 2) * 4;
  // "Landed" barriers, one per chunk modulo this.  A warp that takes every TEAMS-th chunk can tell the two phases of a
  // barrier apart only if it has itself passed the barrier's previous use: TMA loads may land out of order, and with
  // a barrier per stage it could find the phase of a use that another team still waits for.
  static constexpr int FULL_BARS = STAGES * TEAMS;
  static constexpr int NUM_BARS = FULL_BARS + 2 * STAGES + 4;
  static constexpr int SMEM_BYTES = BAR_OFF + NUM_BARS * 8 + 16;
  static constexpr int SMEM_ALLOC = SMEM_BYTES + 1024;
  static constexpr uint32_t TMEM_COLS = 512;
  static constexpr uint32_t A_COL = 256;                       // weights of stage st: columns A_COL + 32 * st, 8 per slab
  static constexpr uint32_t META_COL = A_COL + 32 * STAGES;    // metadata of stage st: META_COL + 4 * st, a column per slab
  static_assert(META_COL % 2 == 0 && META_COL + 4 * STAGES <= TMEM_COLS, "metadata pairs start on even columns");
};

// Token tile class of a work item: N of the instruction = 64 << class.
__device__ __forceinline__ int tile_class(int valid) { return valid <= 64 ? 0 : (valid <= 128 ? 1 : 2); }

__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tc_st4(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// 3-D tiled TMA load of the activation tile: coordinates (K inside a 64-K half, row, 64-K half).
__device__ __forceinline__ void tma_load_3d_hint(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
  return v;
}

// ---- cluster-of-two helpers ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded like mbar_wait; observes arrivals made by the other CTA of the pair.
__device__ __forceinline__ void mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* dead) {
  uint32_t polls = 0;
  while (!mbar_try_wait_cluster(bar, parity)) {
    if ((polls & 15u) == 0 && *dead) return;
    if (++polls > kMaxPolls) {
      *dead = 1;
      atomicExch(&g_device_status, TRB_ERR_TIMEOUT);
      return;
    }
  }
}
// One instruction for both CTAs: M = 256 (128 TMEM lanes in each CTA), half of the N tokens from each
// CTA's shared memory; TMEM addresses and the descriptor are CTA-relative and equal in both.
// `idesc`: D fp32, A and B fp16, K-major, M = 256, N, the sparsity flag (bit 2) and the metadata id (bits 0-1).
__device__ __forceinline__ void tc_mma_sp_f16_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t e_tmem,
                                                   uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.sp.cta_group::2.kind::f16 [%0], [%1], %2, [%5], %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(e_tmem)
      : "memory");
}
// Arrive on the barrier at this shared-memory offset in both CTAs once the pair's MMAs issued so far retire.
// (`mask`: the pair's CTAs by their rank in the cluster).
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar, uint16_t mask = 3) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(mask)
               : "memory");
}

__global__ void __launch_bounds__(TcSpCfg::THREADS, 1)
delta_gemm_tcsp_kernel(const __grid_constant__ CUtensorMap tm_x0, const __grid_constant__ CUtensorMap tm_x1,
                       const __grid_constant__ CUtensorMap tm_x2, const __grid_constant__ CUtensorMap tm_q,
                       const __grid_constant__ CUtensorMap tm_m, const __grid_constant__ CUtensorMap tm_s,
                       const __grid_constant__ GemmArgs a) {
  using Cfg = TcSpCfg;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  int* rows = reinterpret_cast<int*>(smem + Cfg::ROWS_OFF);
  int* prefix = reinterpret_cast<int*>(smem + Cfg::PREFIX_OFF);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);   // [FULL_BARS] TMA data of a chunk landed
  uint64_t* aready_bar = full_bar + Cfg::FULL_BARS;                                // leader: weights + metadata of a stage in TMEM, both CTAs
  uint64_t* empty_bar = aready_bar + STAGES;                               // MMAs of a stage retired
  uint64_t* accready_bar = empty_bar + STAGES;                             // [2] accumulator complete
  uint64_t* accfree_bar = accready_bar + 2;                                // [2] leader: accumulator half drained by both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accfree_bar + 2);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  int n_seg = 0;

  // A tile list that the router left empty (the usual case at decode sizes): leave before anything
  // is set up.  Both CTAs of a pair read the same count.
  pdl_launch_dependents();
  if (a.mode == kSegTiles && a.n_seg_ptr != nullptr) {
    pdl_wait();
    if (*a.n_seg_ptr <= 0) return;
  }

  if (tid == 0) {
    for (int s = 0; s < Cfg::FULL_BARS; ++s) mbar_init(&full_bar[s], 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&aready_bar[s], 4 * Cfg::CTAS);   // the leader's barrier counts both CTAs' warps of a team
      mbar_init(&empty_bar[s], 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&accready_bar[h], 1);
      mbar_init(&accfree_bar[h], Cfg::EPI_WARPS * Cfg::CTAS);
    }
    *dead = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(Cfg::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_wait();   // everything below reads what the kernels launched before this one wrote
  n_seg = a.n_seg_ptr ? *a.n_seg_ptr : a.n_seg;
  n_seg = max(0, min(n_seg, a.mode == kSegTiles ? a.n_seg : kMaxSegments));
  int total_tiles;
  if (a.mode == kSegList) {
    if (warp == 0) {
      int running = 0;
      for (int base = 0; base < n_seg; base += 32) {
        const int s = base + lane;
        int c = 0;
        if (s < n_seg) {
          const int cnt = a.seg_count[s];
          c = cnt > 0 ? (cnt + Cfg::TT - 1) / Cfg::TT : 0;
        }
        int inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += v;
        }
        if (s < n_seg) prefix[s] = running + inc - c;
        running += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) prefix[n_seg] = running;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();     // both CTAs' barriers exist before any remote arrive
  tc_fence_after();
  if (a.mode == kSegList) total_tiles = prefix[n_seg];
  else total_tiles = a.mode == kSegTiles ? n_seg : (a.mode == kSegSingle ? (a.rows + Cfg::TT - 1) / Cfg::TT : a.rows);
  const uint32_t tmem_base = *tmem_slot;

  const int n_stripes = (a.N + Cfg::SW * 64 - 1) / (Cfg::SW * 64);
  const int n_items = total_tiles * n_stripes;
  // Work items go round-robin over CTA pairs: CTA `rank` of a pair owns columns [col0 + 128 * rank, +128)
  // of the item and stages its half of the tile's tokens.
  const uint32_t rank = cluster_ctarank();
  const int item0 = (int)(blockIdx.x >> 1);
  const int item_step = (int)(gridDim.x >> 1);
  const int my_col = (int)rank * 128;
  const int slabs = a.K / 32;
  const int k_chunks = a.K / Cfg::KC;      // K is a multiple of 128
  const uint32_t smem_base = smem_u32(smem);

  if (warp == 0) {
    // ------------------------------ TMA producer: activations ------------------------------
    if (lane == 0) {
      prefetch_tmap(&tm_x0);
      prefetch_tmap(&tm_x1);
      prefetch_tmap(&tm_x2);
      const uint64_t pol_x = policy_evict_last();
      int st = 0, fb = 0;
      uint32_t phase = 0;
      for (int item = item0; item < n_items; item += item_step) {
        const WorkItem w = decode_item<Cfg>(a, prefix, n_seg, n_stripes, item);
        if (!w.ok) continue;
        const int cls = tile_class(w.valid);
        const int half = 32 << cls;            // rows of the tile staged by this CTA
        const CUtensorMap* tm_x = cls == 0 ? &tm_x0 : (cls == 1 ? &tm_x1 : &tm_x2);
        const uint32_t stage_tx = half * Cfg::KC * 2 + Cfg::Q_BYTES + Cfg::M_BYTES + (a.grouped ? Cfg::S_BYTES : 0);
        const int row0 = w.row0 + (int)rank * half;
        for (int kc = 0; kc < k_chunks; ++kc) {
          mbar_wait(&empty_bar[st], phase ^ 1, dead);
          // The stage's one arrival, carrying the bytes of this load and of the weight producer's loads.
          mbar_arrive_expect_tx(&full_bar[fb], stage_tx);
          tma_load_3d_hint(smem + st * Cfg::STAGE_BYTES + Cfg::B_OFF, tm_x, 0, row0, 2 * kc, &full_bar[fb], pol_x);
          if (++st == STAGES) { st = 0; phase ^= 1; }
          if (++fb == Cfg::FULL_BARS) fb = 0;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (rank == 0) {
      const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
      int st = 0;
      uint32_t phase = 0, used[2] = {0, 0};
      int turn = 0;
      for (int item = item0; item < n_items; item += item_step) {
        const WorkItem w = decode_item<Cfg>(a, prefix, n_seg, n_stripes, item);
        if (!w.ok) continue;
        const int cls = __shfl_sync(0xffffffffu, tile_class(w.valid), 0);
        // A 256-token tile takes both halves of the accumulator columns, smaller ones take turns.
        const int h = cls == 2 ? 0 : turn;
        mbar_wait_cluster(&accfree_bar[h], (used[h] & 1) ^ 1, dead);
        ++used[h];
        if (cls == 2) {
          mbar_wait_cluster(&accfree_bar[1], (used[1] & 1) ^ 1, dead);
          ++used[1];
        } else {
          turn ^= 1;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem + h * 128;
        const uint32_t idesc = (1u << 4) | ((uint32_t)(8 << cls) << 17) | ((256u >> 4) << 24) | (1u << 2);   // N = 64 << cls
        const uint32_t khalf = (32u << cls) * 128u >> 4;      // descriptor step to the second 64-K half
        for (int kc = 0; kc < k_chunks; ++kc) {
          // Every decode warp of both CTAs arrives after its own CTA's TMA data landed and its part of
          // the weights and metadata is in TMEM: the one barrier covers both CTAs' operands.
          mbar_wait_cluster(&aready_bar[st], phase, dead);
          tc_fence_after();
          const uint64_t bdesc = tc_smem_desc(smem_base + st * Cfg::STAGE_BYTES + Cfg::B_OFF);
          const uint32_t a_tmem = tmem + Cfg::A_COL + 32 * st;
          const uint32_t e_tmem = tmem + Cfg::META_COL + 4 * st;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < Cfg::SLABS; ++k)   // per instruction: 8 columns of weights, 64 bytes of B, one metadata column
              tc_mma_sp_f16_pair(d_tmem, a_tmem + 8 * k, bdesc + (k >> 1) * khalf + 4 * (k & 1), e_tmem + (k & 2),
                                 idesc | (k & 1), (kc > 0 || k > 0) ? 1u : 0u);
            tc_commit_pair(&empty_bar[st]);
          }
          __syncwarp();
          if (++st == STAGES) { st = 0; phase ^= 1; }
        }
        if (elect_one()) tc_commit_pair(&accready_bar[h]);
        __syncwarp();
      }
    }
  } else if (warp == 2) {
    // ------------------------------ TMA producer: packed weights, metadata, scales ------------------------------
    // A thread of its own: the TMA unit takes the small boxes while the activation box is in flight.
    if (lane == 0) {
      prefetch_tmap(&tm_q);
      prefetch_tmap(&tm_m);
      if (a.grouped) prefetch_tmap(&tm_s);
      const uint64_t pol_w = policy_evict_first();
      int st = 0, fb = 0;
      uint32_t phase = 0;
      for (int item = item0; item < n_items; item += item_step) {
        const WorkItem w = decode_item<Cfg>(a, prefix, n_seg, n_stripes, item);
        if (!w.ok) continue;
        const int col0 = w.col0 + my_col;
        for (int kc = 0; kc < k_chunks; ++kc) {
          mbar_wait(&empty_bar[st], phase ^ 1, dead);
          uint8_t* sbase = smem + st * Cfg::STAGE_BYTES;
          const int wrow = w.delta * slabs + kc * Cfg::SLABS;
          tma_load_2d_hint(sbase + Cfg::Q_OFF, &tm_q, (col0 / 64) * 128, wrow, &full_bar[fb], pol_w);
          tma_load_2d_hint(sbase + Cfg::M_OFF, &tm_m, (col0 / 64) * 64, wrow, &full_bar[fb], pol_w);
          if (a.grouped)
            tma_load_2d_hint(sbase + Cfg::S_OFF, &tm_s, col0, w.delta * k_chunks + kc, &full_bar[fb], pol_w);
          if (++st == STAGES) { st = 0; phase ^= 1; }
          if (++fb == Cfg::FULL_BARS) fb = 0;
        }
      }
    }
  } else if (warp >= Cfg::DECODE0 && warp < Cfg::EPI0) {
    // ------------------------------ decode warps: packed -> weights + metadata in TMEM ------------------------------
    // Lane of quadrant `quad` = feature n = 32 * quad + lane of the CTA's 128: column block cb = n / 64, group
    // g = n / 8 % 8, position j + 4 * hi inside the group.  Its stored pairs m and m + 4 (m = 0..3) of a slab
    // are the low (hi = 0) or the odd (hi = 1) byte pair of weight word (slab, cb, g, m, j).
    const int team = (warp - Cfg::DECODE0) >> 2;
    const int quad = warp & 3;
    const int n = quad * 32 + lane;
    const int j = lane & 3, hi = (lane >> 2) & 1, g = (n >> 3) & 7;
    // Groups g and g + 2 lie on the same banks: half of the lanes read the words of a pair in the other order.
    const bool flip = (g & 2) != 0;
    const uint32_t q_off = Cfg::Q_OFF + (n >> 6) * 512 + g * 64 + j * 4;
    const uint32_t q_first = q_off + (flip ? 16 : 0), q_second = q_off + (flip ? 0 : 16);
    const uint32_t s_off = Cfg::S_OFF + ((n & ~7) + 2 * j + hi) * 2;     // stored scale order inside 8 columns: 0 4 1 5 2 6 3 7
    const int shift = 8 * hi;
    // Metadata cell of TMEM lane n: (row block n / 16, K half n / 8 % 2, row n % 8) = the 16-bit field of that K
    // half for rows r = 16 * (n / 16) + n % 8 (low) and r + 8 (high).  Row r is block r / 64, group mg, position
    // mj + 4 * mhi: its field is the low (mhi = 0) or high half of metadata word
    // 2 * (mj & 1) + 32 * (mj >> 1) + 4 * mg + (K half) of that block; r + 8 is group mg + 1.  Lanes with
    // mj >= 2 fetch the two words in the other order (same banks otherwise).
    const int mr = 16 * (n >> 4) + (n & 7);
    const int mj = mr & 3, mhi = (mr >> 2) & 1, mg = (mr & 63) >> 3;
    const bool mswap = mj >= 2;
    const uint32_t m_off = Cfg::M_OFF + ((mr >> 6) * 64 + 2 * (mj & 1) + 32 * (mj >> 1) + 4 * mg + ((n >> 3) & 1)) * 4;
    const uint32_t m_first = m_off + (mswap ? 16 : 0), m_second = m_off + (mswap ? 0 : 16);
    const uint32_t msel = mswap ? (mhi ? 0x3276u : 0x1054u) : (mhi ? 0x7632u : 0x5410u);
    const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);

    const uint32_t aready_leader = mapa_shared(smem_u32(aready_bar), 0);
    int st = 0, turn = 0, fb = 0;
    uint32_t phase = 0;                  // of the "landed" barriers
    for (int item = item0; item < n_items; item += item_step) {
      const WorkItem w = decode_item<Cfg>(a, prefix, n_seg, n_stripes, item);
      if (!w.ok) continue;
      for (int kc = 0; kc < k_chunks; ++kc) {
        if (turn == team) {
          mbar_wait(&full_bar[fb], phase, dead);
          const uint32_t sb = smem_base + st * Cfg::STAGE_BYTES;
          uint32_t e[Cfg::SLABS];
#pragma unroll
          for (int s = 0; s < Cfg::SLABS; ++s)
            e[s] = __byte_perm(lds32(sb + m_first + s * 512), lds32(sb + m_second + s * 512), msel);
          tc_fence_after();      // the stage's columns were read by MMAs: retired before TMA filled the stage again
          tc_st4(t_lane + Cfg::META_COL + 4 * st, e[0], e[1], e[2], e[3]);
          uint32_t sc = 0;
          if (a.grouped) sc = lds16(sb + s_off) * 0x10001u;
#pragma unroll
          for (int s = 0; s < Cfg::SLABS; ++s) {
            uint32_t q[4], v[8];
#pragma unroll
            for (int p = 0; p < 2; ++p) {
              const uint32_t w0 = lds32(sb + q_first + s * 1024 + p * 32), w1 = lds32(sb + q_second + s * 1024 + p * 32);
              q[2 * p] = flip ? w1 : w0;
              q[2 * p + 1] = flip ? w0 : w1;
            }
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              int4x4_to_half2x2(q[m] >> shift, v[m], v[m + 4]);
              if (a.grouped) {
                v[m] = hmul2_u32(v[m], sc);
                v[m + 4] = hmul2_u32(v[m + 4], sc);
              }
            }
            tc_st8(t_lane + Cfg::A_COL + 32 * st + 8 * s, v);
          }
          tc_wait_st();          // the stage's words have been used by now: no proxy fence before TMA may overwrite them
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(aready_leader + st * 8);
        }
        if (++turn == Cfg::TEAMS) turn = 0;
        if (++st == STAGES) st = 0;
        if (++fb == Cfg::FULL_BARS) { fb = 0; phase ^= 1; }
      }
    }
  } else if (warp >= Cfg::EPI0) {
    // ------------------------------ epilogue warps ------------------------------
    const int ew = warp - Cfg::EPI0;
    const int quad = warp & 3;
    const uint32_t accfree_leader = mapa_shared(smem_u32(accfree_bar), 0);
    uint32_t done[2] = {0, 0};      // tiles published on each accready barrier so far
    int turn = 0;
    for (int item = item0; item < n_items; item += item_step) {
      WorkItem w = decode_item<Cfg>(a, prefix, n_seg, n_stripes, item);
      w.col0 += my_col;
      if (!w.ok) continue;
      const int cls = tile_class(w.valid);
      const int h = cls == 2 ? 0 : turn;
      if (cls != 2) turn ^= 1;
      for (int t = ew * 32 + lane; t < Cfg::TT; t += Cfg::EPI_WARPS * 32) {
        int r = -1;
        if (t < w.valid) {
          r = w.row0 + t;
          if (a.row_map) r = a.row_map[r];
          if (r < 0 || r >= a.rows) r = -1;
        }
        rows[t] = r;
      }
      const int n = w.col0 + quad * 32 + lane;
      float sf = 1.f;
      if (!a.grouped && n < a.N) sf = __half2float(a.scales[(size_t)w.delta * a.N + n]);
      // One warp polls the barrier (a shared-memory access per poll), the others park on the
      // hardware barrier; the wait spans the whole K loop of the item, so the poller backs off.
      if (ew == 0) {
        uint32_t polls = 0;
        while (!mbar_try_wait(&accready_bar[h], done[h] & 1)) {
          __nanosleep(64);
          if ((polls & 15u) == 0 && *dead) break;
          if (++polls > kMaxPolls) {
            *dead = 1;
            atomicExch(&g_device_status, TRB_ERR_TIMEOUT);
            break;
          }
        }
      }
      ++done[h];
      named_bar_sync(4, Cfg::EPI_WARPS * 32);
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + h * 128;
      const int nbatch = max(1, (w.valid + 31) >> 5);
      // The two warps of a quadrant split the 32-token batches: at the accumulator halves for a 256-token
      // tile, evenly otherwise.  Each hands a half back once, when its last batch of it is in registers
      // (at once if it has none): the next item's MMAs may then overwrite it.
      const int grp = ew >> 2;
      const int per = cls == 2 ? 4 : (nbatch + 1) >> 1;
      const int b0 = grp * per, b1 = min(nbatch, b0 + per);
      auto release = [&](int half) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(accfree_leader + half * 8);
      };
      if (cls == 2) release(grp ^ 1);
      const int mine = cls == 2 ? grp : h;
      if (b1 <= b0) release(mine);
      for (int b = b0; b < b1; ++b) {
        uint32_t v[32];
        tc_ld32(taddr + b * 32, v);
        tc_wait_ld();
        if (b == b1 - 1) release(mine);
        // Transpose the 32-token x 32-feature block through a private 2 KiB patch of shared memory, so
        // that a lane stores 8 consecutive features (16 bytes) of one token instead of one feature.
        {
          __half* patch = reinterpret_cast<__half*>(smem + Cfg::XPOSE_OFF + ew * 2048);
#pragma unroll
          for (int c = 0; c < 32; ++c) patch[c * 32 + lane] = __float2half_rn(__uint_as_float(v[c]) * sf);
          __syncwarp();
          const int f8 = (lane & 3) * 8;                    // feature offset of this lane's 16-byte piece
          const int nb = w.col0 + quad * 32 + f8;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int c = i * 8 + (lane >> 2);              // token of the batch
            const int r = rows[b * 32 + c];
            if (r >= 0 && nb < a.N) {
              uint4 o = *reinterpret_cast<const uint4*>(patch + c * 32 + f8);
              uint4* yp = reinterpret_cast<uint4*>(a.y + (size_t)r * a.N + nb);
              if (a.accumulate) {
                const uint4 old = *yp;
                __half2* oh = reinterpret_cast<__half2*>(&o);
                const __half2* ph = reinterpret_cast<const __half2*>(&old);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 x = __half22float2(oh[e]), y2 = __half22float2(ph[e]);
                  oh[e] = __floats2half2_rn(x.x + y2.x, x.y + y2.y);
                }
              }
              *yp = o;
            }
          }
          __syncwarp();
        }
      }
      named_bar_sync(4, Cfg::EPI_WARPS * 32);          // rows[] is rewritten for the next item after this
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // neither CTA leaves, or frees TMEM, while the other may still touch it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Cfg::TMEM_COLS) : "memory");
  }
}

}  // namespace trb
