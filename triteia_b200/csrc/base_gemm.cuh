// Dense fp16 base GEMM of the path, y[T, N] (+)= x[T, K] * W_base[N, K]^T, with the LoRA expand folded
// into the same accumulator: y += V[T, Kv] * B[Kv, N], where V holds every token's rank-r shrink
// result in the column block of its adapter (zero elsewhere) and B is the adapters' expand matrices
// stacked along K (the natural [M, r, N] tensor seen as [M * r, N]).
//
// The reference runs the base product as torch.matmul (a library GEMM) and then adds the LoRA and
// delta parts in separate passes over y (triteia/python/ops/matmul/ldmm.py:72-76, 86-107;
// sbmm.py:90-93; lora.py:5-9).  Here one kernel on the fifth-generation tensor cores produces
// base + LoRA in one TMEM accumulator and writes y once:
//   tcgen05.mma.cta_group::2.kind::f16: two CTAs of a cluster work on one item of 256 output features
//   x one token tile, 128 features each (own A tile, own accumulator: TMEM lanes = features, columns =
//   tokens) and each stages HALF of the token tile, so an SM pulls a third less through TMA per flop
//   than alone -- at 256 decode tokens the product is bound by that intake, not by the tensor pipe or
//   HBM; two accumulators, so the epilogue of one work item overlaps the MMAs of the next;
//   A operand = W_base rows [128 x 64 K] as they lie in memory (K-major, TMA with 128-byte swizzle),
//   for the LoRA chunks = B rows [64 Kv x 128 features] as they lie in memory (MN-major operand);
//   B operand = x (or V) rows [token tile x 64 K], K-major;
//   warp 0: TMA producer (one thread), warp 1: MMA issuer (an elected lane in the pair's leader CTA) and
//   TMEM owner, warps 2-9: epilogue (tcgen05.ld, convert, 32 x 32 transposes through shared memory,
//   16-byte stores or TMA reductions), warp 10: tells the leader when this CTA's stage has landed.
//   Products with few items run in clusters of four or eight CTAs whose pairs share an item along K.
//   No TMA load uses multicast.  Every wait is bounded; a cluster's CTAs meet at a cluster barrier before
//   any of them leaves.
#pragma once

#include "delta_gemm_tcsp.cuh"

namespace trb {

struct BaseCfg {
  static constexpr int KC = 64;             // K per pipeline stage (one 128-byte swizzle atom of fp16)
  static constexpr int STAGES = 6;
  static constexpr int EPI_WARPS = 8;       // two per TMEM lane quadrant: each takes half of the token batches
  static constexpr int THREADS = (3 + EPI_WARPS) * 32;
  static constexpr int MAX_TT = 256;        // largest token tile (UMMA N)
  static constexpr int A_BYTES = 128 * KC * 2;                 // 16 KiB: this CTA's 128 features
  static constexpr int B_BYTES = (MAX_TT / 2) * KC * 2;        // 16 KiB: this CTA's half of the token tile
  static constexpr int A_OFF = 0;
  static constexpr int B_OFF = A_BYTES;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;        // 32 KiB, a multiple of 1 KiB
  static constexpr int XPOSE_OFF = STAGES * STAGE_BYTES;                  // [EPI_WARPS][32 tokens][32 features] halves
  static constexpr int PREFIX_OFF = XPOSE_OFF + EPI_WARPS * 2048;         // int [kMaxSegments + 2]: tiles before each segment
  static constexpr int BAR_OFF = PREFIX_OFF + (kMaxSegments + 2) * 4;
  static constexpr int NUM_BARS = 3 * STAGES + 4;
  static constexpr int SMEM_BYTES = BAR_OFF + NUM_BARS * 8 + 16;
  static constexpr int SMEM_ALLOC = SMEM_BYTES + 1024;
  static constexpr uint32_t TMEM_COLS = 512;
};
static_assert(BaseCfg::STAGE_BYTES % 1024 == 0, "stages keep the 1 KiB alignment of the swizzle atoms");

struct BaseArgs {
  int T, N, K;        // tokens, output features, input features (K % 64 == 0)
  int kv;             // K extent of the LoRA part (0: none); columns of V and rows of B
  int tt;             // token tile: 32, 64, 128 or 256
  int group;          // token tiles that share a pass over the features (see base_item)
  __half* y;          // fp16 or bf16 by `bf16`
  int accumulate;     // y += result instead of y = result
  int bf16;           // operands and output are bfloat16
  int late_wait;      // the kernel just before feeds a later one only: wait for it at the end (see lora_shrink_rows_kernel)
  // Segmented form (seg != nullptr), the SGMV of the LoRA operators: rows [seg[i], seg[i + 1]) of the
  // input [T, seg_k] meet weight i of a stacked tensor [n_seg, seg_k, N] (row-major, so an MN-major
  // operand as it lies in memory).  K is unused, x is the input, the stacked weights come through tm_b.
  const int* seg;
  int n_seg, seg_k;
  int split_pairs;    // K split: CTA pairs (one cluster) that share an item; 0: a pair takes whole items
};

// Order of the work items.  CTA pairs take items round-robin, so the items of one round are neighbours:
// `group` token tiles x (pairs / group) feature stripes.  A round of 74 pairs then touches 8 tiles and 9-10
// stripes of K halves each, 47 MB at K = 5120, where tile-major order touches every stripe: a 13824 x 5120
// weight is 141 MB, more than L2 holds, and came from HBM again for every token tile.
// Measured: 7001 x 5120 x 13824 bf16 base product inside lora_sgmv, the call 1194 -> 1030 us (the kernel 687 us,
// 1.44 PFLOP/s).
constexpr int kTileGroup = 8;
__device__ __forceinline__ void base_item(int item, int n_tiles, int n_stripes, int group, int& tile, int& stripe) {
  if (group == 1) {
    tile = item / n_stripes;
    stripe = item - tile * n_stripes;
    return;
  }
  const int per = group * n_stripes;
  const int grp = item / per, r = item - grp * per;
  const int tiles = min(group, n_tiles - grp * group);
  stripe = r / tiles;
  tile = grp * group + (r - stripe * tiles);
}

// MN-major operand, 128-byte swizzle: a row of the tile is one K index and holds 64 consecutive
// M (feature) elements = 128 bytes; 8 K rows form a 1 KiB group (stride offset), the next 64
// features start `lbo` bytes further (leading offset).
__device__ __forceinline__ uint64_t tc_smem_desc_mn(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Dense kind::f16 for a CTA pair with a run-time instruction descriptor (token tile and operand
// majorness vary): M = 256 (128 TMEM lanes in each CTA), N rows of B split over the two CTAs.
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// A 32-token x 32-feature block of results, one feature per lane, as rows of 32 features in the warp's patch.
__device__ __forceinline__ void base_fill_patch(const BaseArgs& a, __half* patch, const uint32_t (&v)[32], int lane) {
  if (a.bf16) {
    __nv_bfloat16* pb = reinterpret_cast<__nv_bfloat16*>(patch);
#pragma unroll
    for (int c = 0; c < 32; ++c) pb[c * 32 + lane] = __float2bfloat16_rn(__uint_as_float(v[c]));
  } else {
#pragma unroll
    for (int c = 0; c < 32; ++c) patch[c * 32 + lane] = __float2half_rn(__uint_as_float(v[c]));
  }
}
// Adds a box from shared memory to a tensor in global memory, element by element; a bulk group of its own.
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, const void* src, int c0, int c1) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// A 32-token x 32-feature block of results, one feature per lane: convert, transpose through the warp's patch
// of shared memory, store 16-byte pieces of 8 features.  `old`: the pieces' previous values (ADD).
template <bool ADD>
__device__ __forceinline__ void base_store_batch(const BaseArgs& a, __half* patch, const uint32_t (&v)[32], int row0,
                                                 int valid, int col, int b, int lane, const uint4 (&old)[4]) {
  base_fill_patch(a, patch, v, lane);
  __syncwarp();
  const int f8 = (lane & 3) * 8;                      // feature offset of this lane's 16-byte piece
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = i * 8 + (lane >> 2);                // token of the batch
    const int t = b * 32 + c;
    if (t < valid && col + f8 < a.N) {
      uint4 o = *reinterpret_cast<const uint4*>(patch + c * 32 + f8);
      if constexpr (ADD) {
        if (a.bf16) {
          __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
          const __nv_bfloat162* ph = reinterpret_cast<const __nv_bfloat162*>(&old[i]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 p = __bfloat1622float2(oh[e]), q = __bfloat1622float2(ph[e]);
            oh[e] = __floats2bfloat162_rn(p.x + q.x, p.y + q.y);
          }
        } else {
          __half2* oh = reinterpret_cast<__half2*>(&o);
          const __half2* ph = reinterpret_cast<const __half2*>(&old[i]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 p = __half22float2(oh[e]), q = __half22float2(ph[e]);
            oh[e] = __floats2half2_rn(p.x + q.x, p.y + q.y);
          }
        }
      }
      *reinterpret_cast<uint4*>(a.y + (size_t)(row0 + t) * a.N + col + f8) = o;
    }
  }
  __syncwarp();
}

__device__ __forceinline__ void st_cluster_v4(uint32_t cluster_addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(cluster_addr), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}

// One piece of work of a CTA pair: chunks [kc0, kc1) of an item.
struct BaseUnit {
  int item, kc0, kc1;
};

// SPLIT: for products with fewer items than CTA pairs.  The pairs of a cluster share one item along K; when
// every accumulator of the cluster is complete, each pair sends the token batches that another pair finishes
// as fp32 into that pair's shared memory (the stage ring, idle by then) and adds what it receives for its own
// batches in the order of the ranges.  Everything stays inside the cluster: no workspace, no counters.
// ADD: the result is added to y.  A form of its own: with both epilogues in one kernel the plain one was slower
// (7001 x 64 -> 13824 into a fresh y 89 -> 105 us, 8192 x 64 -> 5120 41 -> 49, 300 x 512 x 512 8.4 -> 9.9).
template <bool SPLIT, bool ADD>
__global__ void __launch_bounds__(BaseCfg::THREADS, 1)
base_gemm_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_b,
                 const __grid_constant__ CUtensorMap tm_y, const BaseArgs a) {
  using Cfg = BaseCfg;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  int* prefix = reinterpret_cast<int*>(smem + Cfg::PREFIX_OFF);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);   // this CTA's TMA data of a stage landed
  uint64_t* ready_bar = full_bar + STAGES;                                 // leader: both CTAs' data landed
  uint64_t* empty_bar = ready_bar + STAGES;                                // MMAs of a stage retired
  uint64_t* accready_bar = empty_bar + STAGES;                             // [2] accumulator complete
  uint64_t* accfree_bar = accready_bar + 2;                                // [2] leader: accumulator drained by both
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accfree_bar + 2);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&ready_bar[s], 2);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accready_bar[b], 1);
      mbar_init(&accfree_bar[b], 2 * Cfg::EPI_WARPS);   // every epilogue warp of both CTAs
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
  if (!a.late_wait) pdl_wait();   // x and V may come from the kernels launched just before
  // Only now may the next kernel start: the indexed LoRA kernel reads its inputs without waiting for this one.
  pdl_launch_dependents();
  const int n_seg = a.seg != nullptr ? max(0, min(a.n_seg, kMaxSegments)) : 0;
  if (a.seg != nullptr && warp == 0) {   // token tiles before each segment
    int running = 0;
    for (int base = 0; base < n_seg; base += 32) {
      const int sg = base + lane;
      int c = 0;
      if (sg < n_seg) {
        const int cnt = a.seg[sg + 1] - max(0, a.seg[sg]);
        c = cnt > 0 ? (cnt + a.tt - 1) / a.tt : 0;
      }
      int inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (sg < n_seg) prefix[sg] = running + inc - c;
      running += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) prefix[n_seg] = running;
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();     // the cluster's barriers exist before any remote arrive
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const uint32_t crank = cluster_ctarank();
  const uint32_t rank = crank & 1, leader = crank & ~1u;   // place in the pair, the pair's leader CTA
  const int n_stripes = (a.N + 255) / 256;            // an item: 256 features (128 per CTA) x one token tile
  const int n_tiles = a.seg != nullptr ? prefix[n_seg] : (a.T + a.tt - 1) / a.tt;
  const int n_items = n_tiles * n_stripes;
  // Token tile -> (first row, rows in use, segment).
  auto tile_rows = [&](int tile, int& row0, int& valid, int& sg) {
    if (a.seg == nullptr) {
      sg = 0;
      row0 = tile * a.tt;
      valid = min(a.tt, a.T - row0);
      return;
    }
    int lo = 0, hi = n_seg;  // largest segment with prefix[seg] <= tile
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (prefix[mid] <= tile) lo = mid; else hi = mid;
    }
    sg = lo;
    const int start = max(0, a.seg[sg]), end = min(a.T, a.seg[sg + 1]);
    row0 = start + (tile - prefix[sg]) * a.tt;
    valid = max(0, min(a.tt, end - row0));
  };
  const int item0 = (int)(blockIdx.x >> 1), item_step = (int)(gridDim.x >> 1);
  const int half_tt = a.tt >> 1;                      // tokens of a tile staged by one CTA
  const int kw = a.seg != nullptr ? 0 : a.K / Cfg::KC;                                  // chunks of the base product
  const int kl = ((a.seg != nullptr ? a.seg_k : a.kv) + Cfg::KC - 1) / Cfg::KC;         // MN-major chunks (LoRA)
  const int k_chunks = kw + kl;
  const uint32_t smem_base = smem_u32(smem);
  // The u-th unit of work of this CTA's pair.
  const int part = (int)(crank >> 1), parts = SPLIT ? a.split_pairs : 1;
  auto unit = [&](int u, BaseUnit& w) -> bool {
    if constexpr (SPLIT) {
      w = BaseUnit{(int)blockIdx.x / (2 * parts), part * k_chunks / parts, (part + 1) * k_chunks / parts};
      return u == 0 && w.item < n_items;
    } else {
      w = BaseUnit{item0 + u * item_step, 0, k_chunks};
      return w.item < n_items;
    }
  };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      prefetch_tmap(&tm_x);
      prefetch_tmap(&tm_w);
      if (kl > 0) {
        prefetch_tmap(&tm_v);
        prefetch_tmap(&tm_b);
      }
      // The token tiles of a round share a weight tile, and with up to three token tiles one round reads it: evict-first
      // (300 x 4096 x 11008 51.3 -> 46.8 us, 512: 51.7 -> 47.5, 700: 51.4 -> 49.2); more token tiles come back to it
      // (1024: 78.9 / 78.2, 2048: 139.6 kept, 149.3 evict-first).
      const uint64_t pol_w = n_tiles > 3 ? policy_evict_normal() : policy_evict_first();
      const uint64_t pol_x = policy_evict_last();
      const uint32_t stage_tx = Cfg::A_BYTES + half_tt * Cfg::KC * 2;
      int st = 0;
      uint32_t phase = 0;
      BaseUnit w;
      for (int u = 0; unit(u, w); ++u) {
        int tile, stripe;
        base_item(w.item, n_tiles, n_stripes, a.group, tile, stripe);
        int row0, valid, sg;
        tile_rows(tile, row0, valid, sg);
        row0 += (int)rank * half_tt;
        const int col0 = stripe * 256 + (int)rank * 128;
        const int wrow0 = a.seg != nullptr ? sg * a.seg_k : 0;      // first row of this segment's weight
        const CUtensorMap* tm_in = a.seg != nullptr ? &tm_x : &tm_v;
        for (int kc = w.kc0; kc < w.kc1; ++kc) {
          mbar_wait(&empty_bar[st], phase ^ 1, dead);
          uint8_t* sbase = smem + st * Cfg::STAGE_BYTES;
          mbar_arrive_expect_tx(&full_bar[st], stage_tx);
          if (kc < kw) {
            tma_load_2d_hint(sbase + Cfg::A_OFF, &tm_w, kc * Cfg::KC, col0, &full_bar[st], pol_w);
            tma_load_2d_hint(sbase + Cfg::B_OFF, &tm_x, kc * Cfg::KC, row0, &full_bar[st], pol_x);
          } else {
            const int j = kc - kw;
            // two boxes of [64 K rows x 64 features]: features col0.. and col0 + 64..
            tma_load_2d_hint(sbase + Cfg::A_OFF, &tm_b, col0, wrow0 + j * Cfg::KC, &full_bar[st], pol_x);
            tma_load_2d_hint(sbase + Cfg::A_OFF + 8192, &tm_b, col0 + 64, wrow0 + j * Cfg::KC, &full_bar[st], pol_x);
            tma_load_2d_hint(sbase + Cfg::B_OFF, tm_in, j * Cfg::KC, row0, &full_bar[st], pol_x);
          }
          if (++st == STAGES) { st = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA) ------------------------------
    if (rank == 0) {
      const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
      // D fp32, A and B fp16 / bf16; N = token tile, M = 256; bit 15: A is MN-major (the LoRA chunks)
      const uint32_t fmt = a.bf16 ? 1u : 0u;           // operand format field: 0 = fp16, 1 = bf16
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (((uint32_t)a.tt >> 3) << 17) | ((256u >> 4) << 24);
      const uint32_t idesc_mn = idesc | (1u << 15);
      int st = 0;
      uint32_t phase = 0;
      uint32_t use[2] = {0, 0};
      int local = 0;
      BaseUnit w;
      for (int u = 0; unit(u, w); ++u) {
        const int buf = local & 1;
        mbar_wait_cluster(&accfree_bar[buf], (use[buf] & 1) ^ 1, dead);
        tc_fence_after();
        const uint32_t d_tmem = tmem + buf * Cfg::MAX_TT;
        for (int kc = w.kc0; kc < w.kc1; ++kc) {
          mbar_wait_cluster(&ready_bar[st], phase, dead);
          tc_fence_after();
          const uint32_t sb = smem_base + st * Cfg::STAGE_BYTES;
          const uint64_t bdesc = tc_smem_desc(sb + Cfg::B_OFF);
          if (elect_one()) {
            if (kc < kw) {
              const uint64_t adesc = tc_smem_desc(sb + Cfg::A_OFF);
#pragma unroll
              for (int k = 0; k < Cfg::KC / 16; ++k)   // +32 bytes of K per instruction = +2 in the address field
                tc_mma_f16_pair(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (kc > w.kc0 || k > 0) ? 1u : 0u);
            } else {
#pragma unroll
              for (int k = 0; k < Cfg::KC / 16; ++k) {  // 16 K rows of 128 bytes per instruction
                // 64-feature halves 8 KiB apart, 8-row K groups 1 KiB apart
                const uint64_t adesc = tc_smem_desc_mn(sb + Cfg::A_OFF + k * 2048, 8192, 1024);
                tc_mma_f16_pair(d_tmem, adesc, bdesc + 2 * k, idesc_mn, (kc > w.kc0 || k > 0) ? 1u : 0u);
              }
            }
            tc_commit_pair(&empty_bar[st], (uint16_t)(3u << leader));
          }
          __syncwarp();
          if (++st == STAGES) { st = 0; phase ^= 1; }
        }
        if (elect_one()) tc_commit_pair(&accready_bar[buf], (uint16_t)(3u << leader));
        __syncwarp();
        ++use[buf];
        ++local;
      }
    }
  } else if (warp == 2 + Cfg::EPI_WARPS) {
    // ------------------------------ stage relay: this CTA's data landed -> the leader ------------------------------
    if (lane == 0) {
      const uint32_t ready_leader = mapa_shared(smem_u32(ready_bar), leader);
      int st = 0;
      uint32_t phase = 0;
      BaseUnit w;
      for (int u = 0; unit(u, w); ++u) {
        for (int kc = w.kc0; kc < w.kc1; ++kc) {
          mbar_wait(&full_bar[st], phase, dead);
          mbar_arrive_cluster(ready_leader + st * 8);
          if (++st == STAGES) { st = 0; phase ^= 1; }
        }
      }
    }
  } else {
    // ------------------------------ epilogue warps ------------------------------
    const int ew = warp - 2;
    const int quad = warp & 3;                        // TMEM lanes this warp may touch: 32 * quad .. + 31
    const uint32_t accfree_leader = mapa_shared(smem_u32(accfree_bar), leader);
    __half* patch = reinterpret_cast<__half*>(smem + Cfg::XPOSE_OFF + ew * 2048);
    uint32_t use[2] = {0, 0};
    int local = 0;
    if constexpr (SPLIT) {
      if (ew == 0) mbar_wait(&accready_bar[0], 0, dead);
      named_bar_sync(4, Cfg::EPI_WARPS * 32);
    }
    BaseUnit w;
    for (int u = 0; !SPLIT && unit(u, w); ++u) {
      int tile, stripe;
      base_item(w.item, n_tiles, n_stripes, a.group, tile, stripe);
      int row0, valid, sg;
      tile_rows(tile, row0, valid, sg);
      const int col0 = stripe * 256 + (int)rank * 128;
      const int buf = local & 1;
      // Each warp drains the 32-token batches b0, b0 + 1, ... of its TMEM lane quadrant (two warps share a
      // quadrant and split the batches).  Accumulating into y: a full batch leaves as a TMA reduction of its 32 x 32
      // block, an addition in the type of y in L2 (the same rounding as a load, an addition and a store), so the
      // warp neither reads y nor waits for it.  The batch that the tile ends in is added and stored by its warp, the
      // old values fetched before the accumulator is complete (700 tokens in 64 segments, 32 -> 4096: 32.9 us when they
      // were fetched behind it, 29.0).
      // LoRA expand of 7001 x 64 x 13824 into y (387 MB read and written): 154 us with the old values prefetched into
      // registers and added by the warps, 88 us this way.
      constexpr int MAXB = BaseCfg::MAX_TT / 32 / 2;    // batches per warp
      const int f8 = (lane & 3) * 8;                  // feature offset of this lane's 16-byte piece
      const int nb = col0 + quad * 32 + f8;
      const int nbatch = max(1, (valid + 31) >> 5);
      const int per = (nbatch + 1) >> 1;
      const int b0 = (ew >> 2) * per, b1 = min(nbatch, b0 + per);
      uint4 old[4];
      if constexpr (ADD) {
        const int tail = valid >> 5;                  // the batch of fewer than 32 tokens, if there is one
        const bool mine = tail >= b0 && tail < b1;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = tail * 32 + i * 8 + (lane >> 2);
          old[i] = (mine && t < valid && nb < a.N) ? *reinterpret_cast<const uint4*>(a.y + (size_t)(row0 + t) * a.N + nb)
                                                   : make_uint4(0, 0, 0, 0);
        }
      }
      if (ew == 0) {                                  // one warp polls, the others park on the hardware barrier
        uint32_t polls = 0;
        while (!mbar_try_wait(&accready_bar[buf], use[buf] & 1)) {
          __nanosleep(64);
          if ((polls & 15u) == 0 && *dead) break;
          if (++polls > kMaxPolls) {
            *dead = 1;
            atomicExch(&g_device_status, TRB_ERR_TIMEOUT);
            break;
          }
        }
      }
      named_bar_sync(4, Cfg::EPI_WARPS * 32);
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + buf * Cfg::MAX_TT;
#pragma unroll
      for (int k = 0; k < MAXB; ++k) {
        const int b = b0 + k;
        uint32_t v[32];
        if (b < b1) {
          tc_ld32(taddr + b * 32, v);
          tc_wait_ld();
        }
        // hand the buffer back once per warp and item: after its last batch is in registers, or at
        // once if it has no batch
        if (b == b1 - 1 || (b1 <= b0 && k == 0)) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(accfree_leader + buf * 8);
        }
        if (b >= b1) continue;
        if constexpr (ADD) {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the patch has been read
          __syncwarp();
          if (valid - b * 32 >= 32) {
            base_fill_patch(a, patch, v, lane);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0 && col0 + quad * 32 < a.N) tma_reduce_add_2d(&tm_y, patch, col0 + quad * 32, row0 + b * 32);
            continue;
          }
        }
        base_store_batch<ADD>(a, patch, v, row0, valid, col0 + quad * 32, b, lane, old);
      }
      ++use[buf];
      ++local;
    }
    if constexpr (ADD) {
      if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // reductions performed
    }
  }

  if constexpr (SPLIT) {
    cluster_sync_all();     // every accumulator of the cluster is complete: the stage rings are free
    const bool epi = warp >= 2 && warp < 2 + Cfg::EPI_WARPS;
    const int ew = warp - 2, quad = warp & 3, grp = ew >> 2;
    BaseUnit w;
    unit(0, w);
    int tile, stripe, row0, valid, sg;
    base_item(w.item, n_tiles, n_stripes, a.group, tile, stripe);
    tile_rows(tile, row0, valid, sg);
    const int col0 = stripe * 256 + (int)rank * 128 + quad * 32;
    const int nbatch = (valid + 31) >> 5;
    const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
    // Part p finishes batches [p * nbatch / parts, (p + 1) * nbatch / parts).  A received block: sending part
    // (without one's own), batch inside the slice, lane quadrant, 4 KiB each; 96 KiB at most.
    const uint32_t slice_max = (uint32_t)((nbatch + parts - 1) / parts);
    auto block_at = [&](int sender, int receiver, int in_slice) {
      const uint32_t from = (uint32_t)(sender < receiver ? sender : sender - 1);
      return ((from * slice_max + in_slice) * 4 + quad) * 4096 + lane * 16;
    };
    if (epi) {
      tc_fence_after();
      for (int p = 0; p < parts; ++p) {
        if (p == part) continue;
        const uint32_t dst = mapa_shared(smem_base, (uint32_t)(2 * p) + rank);
        const int lo = p * nbatch / parts, hi = (p + 1) * nbatch / parts;
        for (int b = lo + grp; b < hi; b += 2) {
          uint32_t v[32];
          tc_ld32(taddr + b * 32, v);
          tc_wait_ld();
          const uint32_t at = dst + block_at(part, p, b - lo);
#pragma unroll
          for (int i = 0; i < 8; ++i) st_cluster_v4(at + i * 512, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
      }
    }
    cluster_sync_all();     // every partial sum has arrived
    if (epi) {
      __half* patch = reinterpret_cast<__half*>(smem + Cfg::XPOSE_OFF + ew * 2048);
      const int lo = part * nbatch / parts, hi = (part + 1) * nbatch / parts;
      for (int b = lo + grp; b < hi; b += 2) {
        uint4 old[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = b * 32 + i * 8 + (lane >> 2), col = col0 + (lane & 3) * 8;
          old[i] = make_uint4(0, 0, 0, 0);
          if (ADD && t < valid && col < a.N) old[i] = *reinterpret_cast<const uint4*>(a.y + (size_t)(row0 + t) * a.N + col);
        }
        uint32_t own[32], v[32];
        tc_ld32(taddr + b * 32, own);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0u;
        for (int p = 0; p < parts; ++p) {
          if (p == part) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(own[i]));
          } else {
            const uint32_t at = smem_base + block_at(p, part, b - lo);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const uint4 r = lds128(at + i * 512);
              v[4 * i] = __float_as_uint(__uint_as_float(v[4 * i]) + __uint_as_float(r.x));
              v[4 * i + 1] = __float_as_uint(__uint_as_float(v[4 * i + 1]) + __uint_as_float(r.y));
              v[4 * i + 2] = __float_as_uint(__uint_as_float(v[4 * i + 2]) + __uint_as_float(r.z));
              v[4 * i + 3] = __float_as_uint(__uint_as_float(v[4 * i + 3]) + __uint_as_float(r.w));
            }
          }
        }
        base_store_batch<ADD>(a, patch, v, row0, valid, col0, b, lane, old);
      }
    }
  }

  if (a.late_wait) pdl_wait();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // no CTA leaves, or frees TMEM, while another may still touch it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Cfg::TMEM_COLS) : "memory");
  }
}

// V[t, :] = 0 except columns [id * rank, (id + 1) * rank) = scale * x[t] @ A[id], for id = indices[t]
// in [0, num_adapters); the row stays zero for any other id.  One CTA per token, A [M, h1, rank] in
// its natural layout.  This is the shrink half of the reference's BGMV pair
// (triteia/csrc/ops/bgmv_impl.cuh:15-137) writing straight into the operand of the expand above.
// late_wait: the kernel launched just before (the row gather of a fused call) writes nothing this one reads, and it
// started only after everything that does had finished, so the two overlap; this one still ends after it, which
// keeps the order of the stream for the kernels behind.
constexpr int kShrinkThreads = 512;

template <class IdxT>
__global__ void __launch_bounds__(kShrinkThreads) lora_shrink_rows_kernel(__half* __restrict__ V, const __half* __restrict__ X,
                                                               const __half* __restrict__ A,
                                                               const IdxT* __restrict__ indices, int h1, int rank,
                                                               int num_adapters, int v_cols, float scale,
                                                               int late_wait) {
  constexpr int WARPS = kShrinkThreads / 32;
  __shared__ float part[WARPS][64];
  const int b = blockIdx.x;
  pdl_launch_dependents();
  if (!late_wait) pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint4* vrow = reinterpret_cast<uint4*>(V + (int64_t)b * v_cols);
  const long long idx = (long long)indices[b];
  const bool has = idx >= 0 && idx < num_adapters;
  const int lo8 = has ? (int)idx * rank / 8 : -1, hi8 = has ? lo8 + rank / 8 : -1;
  for (int i = tid; i < v_cols / 8; i += kShrinkThreads)
    if (i < lo8 || i >= hi8) vrow[i] = make_uint4(0, 0, 0, 0);
  if (!has) {
    if (late_wait) pdl_wait();
    return;
  }
  const __half* am = A + idx * (int64_t)h1 * rank;
  const __half* x = X + (int64_t)b * h1;
  // A row of A holds rank halves = rv 16-byte pieces.  `pw` lanes (rv rounded up to a power of two)
  // share a row, so a warp load covers 32 / pw consecutive rows: contiguous memory, 8 accumulators
  // per lane.
  const int rv = rank / 8;
  const int pw = rv <= 1 ? 1 : (rv <= 2 ? 2 : (rv <= 4 ? 4 : 8));
  const int sub = lane & (pw - 1), rl = lane / pw, rows_per_warp = 32 / pw;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  if (sub < rv) {
#pragma unroll 8
    for (int k = warp * rows_per_warp + rl; k < h1; k += WARPS * rows_per_warp) {
      const float xk = __half2float(x[k]);
      const uint4 wv = *reinterpret_cast<const uint4*>(am + (int64_t)k * rank + sub * 8);
      const uint32_t* pwv = reinterpret_cast<const uint32_t*>(&wv);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&pwv[e]));
        acc[2 * e] = fmaf(xk, f.x, acc[2 * e]);
        acc[2 * e + 1] = fmaf(xk, f.y, acc[2 * e + 1]);
      }
    }
  }
  // lanes with the same `sub` hold partial sums of the same 8 columns
  for (int o = pw; o < 32; o <<= 1)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
  if (lane < pw && sub < rv)
#pragma unroll
    for (int e = 0; e < 8; ++e) part[warp][sub * 8 + e] = acc[e];
  __syncthreads();
  if (tid < rank) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) s += part[w][tid];
    V[(int64_t)b * v_cols + idx * rank + tid] = __float2half_rn(s * scale);
  }
  if (late_wait) pdl_wait();
}

static_assert(BaseCfg::SMEM_ALLOC <= 232448, "shared memory budget of one sm_100 CTA");

// Clusters of 2 * pairs CTAs that the device holds at once (asked once per device and cluster size).
static int max_split_clusters(int dev, int pairs) {
  static std::atomic<int> cached[64][8];
  if (dev < 0 || dev >= 64 || pairs < 1 || pairs >= 8) return 0;
  int v = cached[dev][pairs].load(std::memory_order_relaxed);
  if (v == 0) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(2 * pairs);
    lc.blockDim = dim3(BaseCfg::THREADS);
    lc.dynamicSmemBytes = BaseCfg::SMEM_ALLOC;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2 * pairs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, base_gemm_kernel<true, false>, &lc) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    v = n + 1;
    cached[dev][pairs].store(v, std::memory_order_relaxed);
  }
  return v - 1;
}

// CTA pairs that share an item of a product with `items` items of `k_chunks` chunks: four or two, when all clusters
// run in one round and a pair is spared at least kSplitSaved chunks; otherwise 0.  The exchange costs about 2.4 us, a
// chunk 0.15 (narrow token tiles) to 0.27.
// Measured (device time of a call behind an L2 flush; whole items -> split): 100 x 2048 x 2048 12.6 -> 10.8 us,
// 32 x 4096 x 4096 19.8 -> 15.6, 512 x 4096 x 4096 26.7 -> 22.5, 64 x 3072 x 3072 16.5 -> 12.4; about the line
// 64 x 1536 x 1536 10.3 -> 10.0, 512 x 2048 x 4096 (two pairs) 16.7 -> 16.5; below it, where items stay whole,
// 64 x 512 x 512 6.1 -> 6.9, 100 x 768 x 3072 8.2 -> 9.5, 64 x 1024 x 4096 8.5 -> 9.3, 512 x 1024 x 4096 12.3 -> 13.3.
// Three pairs on two items, which would use the pairs that 43 items leave idle, lost: 256 x 4096 x 11008
// 34.8 -> 38.9, 256 x 2048 x 9216 23.4 -> 31.5.
constexpr int kSplitSaved = 16;
static int choose_split(int dev, long long items, int k_chunks) {
  for (int p = 4; p >= 2; p -= 2)
    if (k_chunks - k_chunks / p >= kSplitSaved && items <= max_split_clusters(dev, p)) return p;
  return 0;
}

static int base_gemm_launch_args(BaseArgs a, const CUtensorMap& tx, const CUtensorMap& tw, const CUtensorMap& tv,
                                 const CUtensorMap& tb, long long items, int dev, cudaStream_t stream) {
  static std::atomic<bool> attr_set[4][64];
  if (!ensure_smem_attr(base_gemm_kernel<false, false>, dev, BaseCfg::SMEM_ALLOC, attr_set[0]) ||
      !ensure_smem_attr(base_gemm_kernel<false, true>, dev, BaseCfg::SMEM_ALLOC, attr_set[1]) ||
      !ensure_smem_attr(base_gemm_kernel<true, false>, dev, BaseCfg::SMEM_ALLOC, attr_set[2]) ||
      !ensure_smem_attr(base_gemm_kernel<true, true>, dev, BaseCfg::SMEM_ALLOC, attr_set[3]))
    return TRB_ERR_CUDA;
  int pairs = sm_count(dev) / 2;
  if (pairs < 1) pairs = 1;
  if (items < pairs) pairs = (int)(items > 0 ? items : 1);
  int cluster = 2;
  if (a.seg == nullptr) a.split_pairs = choose_split(dev, items, a.K / BaseCfg::KC + (a.kv + BaseCfg::KC - 1) / BaseCfg::KC);
  if (a.split_pairs > 0) {
    cluster = 2 * a.split_pairs;
    pairs = a.split_pairs * (int)items;
  }
  CUtensorMap ty = tx;     // used with accumulate only
  if (a.accumulate && !make_map_2d(&ty, a.bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.y,
                                   (uint64_t)a.T, (uint64_t)a.N, 32, 32, CU_TENSOR_MAP_SWIZZLE_NONE))
    return TRB_ERR_CUDA;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(2 * pairs);
  lc.blockDim = dim3(BaseCfg::THREADS);
  lc.dynamicSmemBytes = BaseCfg::SMEM_ALLOC;
  lc.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // the kernel waits (pdl_wait) before it reads
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = 2;
  auto kernel = a.split_pairs > 0 ? (a.accumulate ? base_gemm_kernel<true, true> : base_gemm_kernel<true, false>)
                                  : (a.accumulate ? base_gemm_kernel<false, true> : base_gemm_kernel<false, false>);
  return cudaLaunchKernelEx(&lc, kernel, tx, tw, tv, tb, ty, a) == cudaSuccess ? TRB_OK : TRB_ERR_CUDA;
}

static int token_tile_for(int rows) { return rows <= 32 ? 32 : rows <= 64 ? 64 : rows <= 128 ? 128 : 256; }

static int base_gemm_launch(const void* x, const void* w, void* y, int T, int N, int K, const void* v, const void* b,
                            int kv, int accumulate, int bf16, int dev, cudaStream_t stream, int late_wait = 0) {
  BaseArgs a{};
  a.late_wait = late_wait;
  a.T = T; a.N = N; a.K = K; a.kv = kv;
  a.tt = token_tile_for(T);
  a.group = kTileGroup;
  a.y = (__half*)y;
  a.accumulate = accumulate;
  a.bf16 = bf16;
  const CUtensorMapDataType dt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tx, tw, tv, tb;
  if (!make_map_2d(&tx, dt, 2, x, (uint64_t)T, (uint64_t)K, a.tt / 2, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return TRB_ERR_CUDA;
  if (!make_map_2d(&tw, dt, 2, w, (uint64_t)N, (uint64_t)K, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return TRB_ERR_CUDA;
  if (kv > 0) {
    if (!make_map_2d(&tv, dt, 2, v, (uint64_t)T, (uint64_t)kv, a.tt / 2, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return TRB_ERR_CUDA;
    if (!make_map_2d(&tb, dt, 2, b, (uint64_t)kv, (uint64_t)N, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return TRB_ERR_CUDA;
  } else {
    tv = tx;   // never dereferenced
    tb = tw;
  }
  const long long items = (long long)((T + a.tt - 1) / a.tt) * ((N + 255) / 256);   // one item per CTA pair
  return base_gemm_launch_args(a, tx, tw, tv, tb, items, dev, stream);
}

// Token tile of the segmented form: the smallest whose items still run in one round (a round of narrow tiles streams
// the input over all SMs: LoRA shrink, one stripe), otherwise the widest that the longest segment fills.
// Measured (device time of a shrink behind an L2 flush, widest tile -> this): 7001 tokens in 16 segments, 5120 -> 64,
// 36.9 -> 33.1 us; 700 in 64, 4096 -> 32, 26.4 -> 22.5; 2000 in 4, 2048 -> 32, 15.1 -> 13.2.
static int segment_tile_for(int rows, int T, int n_seg, int n_stripes, int dev) {
  const int widest = token_tile_for(rows);
  for (int tt = 32; tt < widest; tt *= 2)
    if (((long long)T / tt + n_seg) * n_stripes <= sm_count(dev) / 2) return tt;
  return widest;
}

// Segmented form: y[seg[i] : seg[i + 1]] (+)= x[same rows] @ w[i], w stacked [n_seg, d_in, d_out].
static int sgmv_stacked_launch(void* y, const void* x, const void* w, const int* seg, int n_seg, int T, int d_in,
                               int d_out, int max_rows, int accumulate, int bf16, int dev, cudaStream_t stream) {
  BaseArgs a{};
  a.T = T; a.N = d_out; a.K = 0; a.kv = 0;
  a.tt = segment_tile_for(max_rows > 0 ? max_rows : T, T, n_seg, (d_out + 255) / 256, dev);
  // Tile after tile: the stacked weights of LoRA stay in L2, and with few chunks per item the grouped order only cost
  // (grouped -> this, device time: 2000 tokens in 4 segments, 32 -> 2048, 10.4 -> 8.8 us; 8192 in 16, 64 -> 5120, 45.1 ->
  // 41.1; 700 in 64, 32 -> 4096 added to y, 28.7 -> 27.6).
  a.group = 1;
  a.y = (__half*)y;
  a.accumulate = accumulate;
  a.bf16 = bf16;
  a.seg = seg; a.n_seg = n_seg; a.seg_k = d_in;
  const CUtensorMapDataType dt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tx, tb;
  if (!make_map_2d(&tx, dt, 2, x, (uint64_t)T, (uint64_t)d_in, a.tt / 2, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return TRB_ERR_CUDA;
  if (!make_map_2d(&tb, dt, 2, w, (uint64_t)n_seg * d_in, (uint64_t)d_out, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B))
    return TRB_ERR_CUDA;
  const long long items = ((long long)T / a.tt + n_seg) * ((d_out + 255) / 256);     // upper bound: the lengths are on the device
  return base_gemm_launch_args(a, tx, tx, tx, tb, items, dev, stream);
}

template <class IdxT>
static int lora_shrink_rows_launch(void* v, const void* x, const void* wa, const void* indices, int batch, int h1, int rank,
                                   int num_adapters, int v_cols, float scale, int late_wait, cudaStream_t stream) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(batch);
  lc.blockDim = dim3(kShrinkThreads);
  lc.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, lora_shrink_rows_kernel<IdxT>, (__half*)v, (const __half*)x, (const __half*)wa,
                            (const IdxT*)indices, h1, rank, num_adapters, v_cols, scale, late_wait) == cudaSuccess
             ? TRB_OK
             : TRB_ERR_CUDA;
}

}  // namespace trb

extern "C" int trb_base_gemm(const void* x, const void* base_weight, void* y, int num_tokens, int prob_m, int prob_k,
                             const void* lora_v, const void* lora_b, int lora_k, int accumulate, int dtype, int dev,
                             void* stream) {
  using namespace trb;
  if (num_tokens < 0 || prob_m < 0 || prob_k < 0 || lora_k < 0) return TRB_ERR_BAD_ARG;
  if (num_tokens == 0 || prob_m == 0) return TRB_OK;
  if (!x || !base_weight || !y || (lora_k > 0 && (!lora_v || !lora_b))) return TRB_ERR_BAD_ARG;
  if (prob_k == 0 || prob_k % 64 != 0 || prob_m % 8 != 0 || lora_k % 8 != 0) return TRB_ERR_PROB_SHAPE;
  if (dtype != TRB_F16 && dtype != TRB_BF16) return TRB_ERR_KERN_SHAPE;
  const uintptr_t bits = (uintptr_t)x | (uintptr_t)base_weight | (uintptr_t)y | (uintptr_t)lora_v | (uintptr_t)lora_b;
  if (bits & 15) return TRB_ERR_BAD_ARG;
  if (cudaSetDevice(dev) != cudaSuccess) return TRB_ERR_CUDA;
  return base_gemm_launch(x, base_weight, y, num_tokens, prob_m, prob_k, lora_v, lora_b, lora_k, accumulate ? 1 : 0,
                          dtype == TRB_BF16, dev, (cudaStream_t)stream);
}

extern "C" int trb_base_lora(const void* x, const void* base_weight, void* y, const void* wa, const void* wb,
                             const void* indices, int index_is_64bit, int num_tokens, int prob_m, int prob_k, int rank,
                             int num_adapters, float scale, int dtype, int dev, void* stream) {
  using namespace trb;
  const int r = trb_base_gemm(x, base_weight, y, num_tokens, prob_m, prob_k, nullptr, nullptr, 0, 0, dtype, dev, stream);
  if (r != TRB_OK) return r;
  return lora_indexed_call(y, x, wa, wb, indices, index_is_64bit, num_tokens, prob_k, prob_m, rank, num_adapters, scale, dtype,
                           dev, 1, (cudaStream_t)stream);
}

extern "C" int trb_sgmv_stacked(void* y, const void* x, const void* w, const void* s, int num_problems, int num_rows,
                                int d_in, int d_out, int max_rows, int accumulate, int dtype, int dev, void* stream) {
  using namespace trb;
  if (num_problems == 0 || num_rows == 0) return TRB_OK;
  if (num_problems < 0 || num_rows < 0 || !y || !x || !w || !s) return TRB_ERR_BAD_ARG;
  if (d_in <= 0 || d_out <= 0 || d_in % 8 != 0 || d_out % 8 != 0 || num_problems > kMaxSegments) return TRB_ERR_KERN_SHAPE;
  if ((long long)num_problems * d_in >= (1ll << 31)) return TRB_ERR_KERN_SHAPE;
  if (dtype != TRB_F16 && dtype != TRB_BF16) return TRB_ERR_KERN_SHAPE;
  if (((uintptr_t)x | (uintptr_t)y | (uintptr_t)w) & 15) return TRB_ERR_BAD_ARG;
  if (cudaSetDevice(dev) != cudaSuccess) return TRB_ERR_CUDA;
  return sgmv_stacked_launch(y, x, w, (const int*)s, num_problems, num_rows, d_in, d_out, max_rows, accumulate ? 1 : 0,
                             dtype == TRB_BF16, dev, (cudaStream_t)stream);
}

extern "C" int trb_lora_shrink_rows(void* v, const void* x, const void* wa, const void* indices, int index_is_64bit,
                                    int batch, int h1, int rank, int num_adapters, int v_cols, float scale, int dev,
                                    void* stream) {
  using namespace trb;
  if (batch == 0) return TRB_OK;
  if (batch < 0 || num_adapters <= 0 || !v || !x || !wa || !indices) return TRB_ERR_BAD_ARG;
  if (rank <= 0 || rank > 64 || rank % 8 != 0 || h1 <= 0 || v_cols % 8 != 0 || (long long)num_adapters * rank > v_cols)
    return TRB_ERR_KERN_SHAPE;
  if (((uintptr_t)v | (uintptr_t)wa) & 15) return TRB_ERR_BAD_ARG;
  if (cudaSetDevice(dev) != cudaSuccess) return TRB_ERR_CUDA;
  cudaStream_t st = (cudaStream_t)stream;
  return index_is_64bit
             ? lora_shrink_rows_launch<int64_t>(v, x, wa, indices, batch, h1, rank, num_adapters, v_cols, scale, 0, st)
             : lora_shrink_rows_launch<int32_t>(v, x, wa, indices, batch, h1, rank, num_adapters, v_cols, scale, 0, st);
}

// One call for base product + (LoRA adapter or packed delta) per token: router and row gather of the delta part
// first, the LoRA shrink (or, without adapters, the base product) overlapping them, then base product and LoRA
// expand into y, then the grouped delta kernels adding into y.  The order lets the small kernels run beside the large
// ones on one stream, without a second stream, events or a host call per kernel.
extern "C" int trb_base_indexed(const void* x, const void* base_weight, const void* wa, const void* wb, const void* qweights,
                                const void* metas, const void* scales, const void* indices, void* y, void* v, int num_tokens,
                                int prob_m, int prob_k, int num_adapters, int rank, int num_deltas, int groupsize,
                                void* scratch, size_t scratch_bytes, int dev, void* stream_v) {
  using namespace trb;
  if (num_tokens < 0 || prob_m < 0 || prob_k < 0 || num_adapters < 0 || num_deltas <= 0) return TRB_ERR_BAD_ARG;
  if (num_tokens == 0 || prob_m == 0) return TRB_OK;
  if (!x || !base_weight || !y || !indices || !scratch || (num_adapters > 0 && (!wa || !wb || !v))) return TRB_ERR_BAD_ARG;
  if (prob_k == 0 || prob_k % 64 != 0 || prob_m % 8 != 0) return TRB_ERR_PROB_SHAPE;
  if (num_adapters > 0 && (rank <= 0 || rank > 64 || rank % 8 != 0)) return TRB_ERR_KERN_SHAPE;
  if (((uintptr_t)x | (uintptr_t)base_weight | (uintptr_t)y | (uintptr_t)wa | (uintptr_t)wb | (uintptr_t)v) & 15) return TRB_ERR_BAD_ARG;
  const int v_cols = num_adapters * rank;
  cudaStream_t stream = (cudaStream_t)stream_v;
  RouteSrc src{};
  src.indices = (const int*)indices;
  src.id_offset = num_adapters;
  auto delta = [&](int phase) {
    return sbmm_indexed_impl(x, qweights, metas, scales, src, y, num_tokens, prob_m, prob_k, num_deltas, groupsize, 1, scratch,
                             scratch_bytes, dev, stream, nullptr, 0, phase);
  };
  int r = delta(1);
  if (r == TRB_OK && num_adapters > 0)
    r = lora_shrink_rows_launch<int32_t>(v, x, wa, indices, num_tokens, prob_k, rank, num_adapters, v_cols, 1.f, 1, stream);
  if (r == TRB_OK)
    r = base_gemm_launch(x, base_weight, y, num_tokens, prob_m, prob_k, num_adapters > 0 ? v : nullptr,
                         num_adapters > 0 ? wb : nullptr, v_cols, 0, 0, dev, stream, num_adapters > 0 ? 0 : 1);
  if (r == TRB_OK) r = delta(2);
  return r;
}
