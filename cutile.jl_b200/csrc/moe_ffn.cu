// Mixture-of-experts FFN on one GPU (cutile_moe, examples/moe.jl:218-257) in four kernels:
//   moe_sort_gather_kernel  sorts the (token, choice) slots by expert and copies the token rows into that order, every
//                           expert's rows padded to a multiple of 16;
//   moe_pair_gemm_kernel    gate/up projection with SwiGLU, then the down projection scaled by the routing weight, both on
//                           sorted rows, results again in sorted order;
//   moe_sorted_combine_kernel  sum over the top-k slots of a token (:256).
//
// With few tokens the whole is bound by streaming the chosen experts' weights once (403 MB at 256 tokens, top-2 over 32
// experts), with many by the tensor cores.  A kernel that gathers its token rows itself pays for it in every k-block; the
// copy is 2 x 8192 rows x 2 KB at 4096 tokens and lets both projections take all operands as plain TMA tiles.
//
// The weights are the M operand of the MMA: a CTA pair (cta_group::2) takes 256 weight rows, the slots of one block of an
// expert are the N operand, so a block costs what it holds, rounded up to 16 slots.  With the slots as M (128 or 256 rows
// whatever the block holds) 4096 tokens cost 25 % (50 % in pairs) of padding.  An expert with more than 256 slots is cut
// into equal blocks.
#include <math.h>

#include <algorithm>

#include "ctx.h"
#include "ptx.cuh"

using namespace ctb;
using namespace ctb_internal;

namespace {

constexpr int kMaxExperts = 256;
constexpr int kMaxBlockSlots = 256;  // MMA N

// ------------------------------------------------------------------ sort and gather
constexpr int kSortThreads = 512, kSortWarps = kSortThreads / 32, kSortCtas = 148;
constexpr int kSortLocal = 16384;  // up to this many slots every CTA counts all of them itself

struct Block {  // slots of one expert that one GEMM item takes
  int expert, row0, n, pad;
};
struct SortParams {
  const __half* topk_w;  // (T, topk) column-major like the ids
  const uint4* X;
  uint4* xs;        // rows in sorted order
  int* pos_of;      // sorted row of flat slot token * topk + choice
  float* wts;       // routing weight of a sorted row
  Block* table;
  int* num_blocks;  // [0] blocks, [1] slots of the largest
  const int* counts;  // [kSortCtas][E + 1]: slots per expert in every CTA's chunk, then 1 if an id is out of range; or null
  const unsigned char* warm;  // gate/up weights, for the L2 (null: not)
  long long warm_expert;      // bytes of one expert's gate or up rows
  int warm_tile, warm_mtiles;  // bytes of the 64 rows that a CTA of an item streams; row tiles per block
  int T, topk, E, vecs, total, chunk;
  int* status;
};

// Mask of the lanes of the (converged) warp that hold the same value v (`bits` bits; lanes with v < 0 form a group).
__device__ __forceinline__ unsigned same_value(int v, int bits) {
  unsigned m = __ballot_sync(0xffffffffu, v < 0);
  m = v < 0 ? m : ~m;
  for (int b = 0; b < bits; ++b) {
    const unsigned bal = __ballot_sync(0xffffffffu, (v >> b) & 1);
    m &= ((v >> b) & 1) ? bal : ~bal;
  }
  return m;
}

// Slots per expert of one CTA's chunk (only for more slots than kSortLocal).
template <typename IdT>
__global__ void __launch_bounds__(kSortThreads)
    moe_count_kernel(const IdT* __restrict__ ids, int T, int topk, int E, int total, int chunk, int* __restrict__ counts) {
  grid_dependency_sync();
  __shared__ int cnt[kMaxExperts + 1];
  for (int e = threadIdx.x; e <= E; e += kSortThreads) cnt[e] = 0;
  __syncthreads();
  const int lo = min(total, (int)blockIdx.x * chunk), hi = min(total, lo + chunk);
  for (int i = lo + threadIdx.x; i < hi; i += kSortThreads) {
    const int tok = i / topk, slot = i - tok * topk;
    const long long e = (long long)ids[(long long)slot * T + tok] - 1;
    if (e >= 0 && e < E) atomicAdd(&cnt[e], 1);
    else cnt[E] = 1;
  }
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += kSortThreads) counts[blockIdx.x * (E + 1) + e] = cnt[e];
}

// CTA c places the flat slots [c * chunk, (c + 1) * chunk) and copies their rows.  Nothing is exchanged between the CTAs:
// each counts all slots (or reads the chunks' counts) and so knows where every expert's rows and its own share of them
// start; the order inside an expert is the flat slot order, as in moe_align_tile_size (examples/moe.jl:142-183).
// A chain of latencies (7.9 us at 512 slots by itself).  While the rows are copied the L2 fetches the weights that the
// GEMM's CTAs stream first.
template <typename IdT>
__global__ void __launch_bounds__(kSortThreads) moe_sort_gather_kernel(const IdT* __restrict__ ids, const SortParams p) {
  extern __shared__ int sort_smem[];  // small, so that the next kernel's CTAs fit beside
  __shared__ int spos[kSortThreads];
  __shared__ int bad, nmax;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, E = p.E, cta = blockIdx.x;
  int *tot = sort_smem, *base = tot + E, *wcount = base + E, *bstart = wcount + kSortWarps * E;  // [E], [E], [warps][E], [E + 1]
  for (int e = tid; e < E; e += kSortThreads) tot[e] = base[e] = 0;
  if (tid == 0) bad = nmax = 0;
  __syncthreads();
  grid_dependency_sync();
  const int lo = min(p.total, cta * p.chunk), hi = min(p.total, lo + p.chunk);
  // ---- slots per expert: all of them, and those before this CTA's
  if (!p.counts) {
    for (int slot = 0; slot < p.topk; ++slot) {
      const IdT* col = ids + (long long)slot * p.T;
      for (int t0 = tid; t0 < p.T; t0 += 8 * kSortThreads) {
        long long e[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) e[q] = t0 + q * kSortThreads < p.T ? (long long)col[t0 + q * kSortThreads] - 1 : 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (t0 + q * kSortThreads >= p.T) continue;
          if (e[q] < 0 || e[q] >= E) {
            bad = 1;
          } else {
            atomicAdd(&tot[e[q]], 1);
            if ((t0 + q * kSortThreads) * p.topk + slot < lo) atomicAdd(&base[e[q]], 1);
          }
        }
      }
    }
  } else {
    for (int e = tid; e <= E; e += kSortThreads) {
      int all = 0, before = 0;
#pragma unroll 8
      for (int c = 0; c < kSortCtas; ++c) {
        const int n = __ldcg(p.counts + c * (E + 1) + e);
        all += n;
        before += c < cta ? n : 0;
      }
      if (e < E) {
        tot[e] = all;
        base[e] = before;
      } else if (all) {
        bad = 1;
      }
    }
  }
  __syncthreads();
  if (bad) {  // reported, and no expert runs; the combine kernel finds valid positions
    if (cta == 0 && tid == 0) {
      atomicMax(p.status, DEV_BAD_INDEX);
      p.num_blocks[0] = 0;
      p.num_blocks[1] = 16;
    }
    for (int i = lo + tid; i < hi; i += kSortThreads) p.pos_of[i] = 0;
    return;
  }
  // ---- first row and first block of every expert
  if (warp == 0) {
    int rows = 0, blocks = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane, c = e < E ? tot[e] : 0, padded = (c + 15) & ~15, nb = (c + kMaxBlockSlots - 1) / kMaxBlockSlots;
      int r = padded, b = nb;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int rr = __shfl_up_sync(0xffffffffu, r, o), bb = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) { r += rr; b += bb; }
      }
      if (e < E) {
        base[e] += rows + r - padded;
        bstart[e] = blocks + b - nb;
      }
      rows += __shfl_sync(0xffffffffu, r, 31);
      blocks += __shfl_sync(0xffffffffu, b, 31);
    }
    if (lane == 0) bstart[E] = blocks;
  }
  __syncthreads();
  // ---- weights that this CTA's part of the first gate/up item streams
  if (p.warm) {
    const int item = cta >> 1, b = item / p.warm_mtiles;
    if (b < bstart[E]) {
      int l = 0, h = E - 1;  // last expert whose first block is <= b
      while (l < h) {
        const int mid = (l + h + 1) >> 1;
        if (bstart[mid] <= b) l = mid;
        else h = mid - 1;
      }
      const long long first = ((long long)(item - b * p.warm_mtiles) * 2 + (cta & 1)) * p.warm_tile;
      const unsigned char* gate = p.warm + (long long)l * 2 * p.warm_expert + first;
      for (int x = tid * 128; x < min((long long)p.warm_tile, p.warm_expert - first); x += kSortThreads * 128) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(gate + x) : "memory");
        asm volatile("prefetch.global.L2 [%0];" ::"l"(gate + p.warm_expert + x) : "memory");
      }
    }
  }
  if (cta == 0) {  // the block table; this CTA has no slots before it: base is the experts' first row
    for (int e = tid; e < E; e += kSortThreads) {
      const int c = tot[e], nb = bstart[e + 1] - bstart[e];
      if (!nb) continue;
      const int size = ((c + nb - 1) / nb + 15) & ~15;
      for (int k = 0; k < nb; ++k) {
        const int n = (min(size, c - k * size) + 15) & ~15;
        p.table[bstart[e] + k] = {e, base[e] + k * size, max(n, 16), 0};
      }
      atomicMax(&nmax, size);
    }
    __syncthreads();
    if (tid == 0) {
      p.num_blocks[0] = bstart[E];
      p.num_blocks[1] = nmax;
    }
    __syncthreads();
  }
  // ---- this CTA's slots, kSortThreads at a time: stable positions, then the rows
  int ebits = 1;
  while ((1 << ebits) < E) ++ebits;
  for (int b0 = lo; b0 < hi; b0 += kSortThreads) {
    for (int i = tid; i < kSortWarps * E; i += kSortThreads) wcount[i] = 0;
    __syncthreads();
    const int i = b0 + tid;
    int e = -1, tok = 0, slot = 0;
    if (i < hi) {
      tok = i / p.topk;
      slot = i - tok * p.topk;
      e = (int)ids[(long long)slot * p.T + tok] - 1;
    }
    const unsigned grp = same_value(e, ebits);
    const int rank = __popc(grp & ((1u << lane) - 1));
    if (e >= 0 && rank == 0) wcount[warp * E + e] = __popc(grp);
    __syncthreads();
    if (tid < E) {
      int run = base[tid];
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) {
        const int c = wcount[w * E + tid];
        wcount[w * E + tid] = run;
        run += c;
      }
      base[tid] = run;
    }
    __syncthreads();
    if (e >= 0) {
      const int pos = wcount[warp * E + e] + rank;
      spos[tid] = pos;
      p.pos_of[i] = pos;
      p.wts[pos] = __half2float(p.topk_w[(long long)slot * p.T + tok]);
    }
    __syncthreads();
    const int n = min(kSortThreads, hi - b0) * p.vecs;
    for (int x0 = tid; x0 < n; x0 += 8 * kSortThreads) {
      uint4 v[8];
      long long to[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int x = x0 + q * kSortThreads;
        if (x < n) {
          const int r = x / p.vecs, c = x - r * p.vecs;
          v[q] = __ldg(p.X + (long long)((b0 + r) / p.topk) * p.vecs + c);
          to[q] = (long long)spos[r] * p.vecs + c;
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (x0 + q * kSortThreads < n) p.xs[to[q]] = v[q];
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ the two projections
constexpr int kBK = 64;                      // K elements per stage (128 bytes)
constexpr int kABytes = 128 * kBK * 2;       // a CTA's 128 weight rows of a k-block
constexpr int kMaxStages = 12;
constexpr int kRingBytes = 192 * 1024;
constexpr int kEpiWarps = 8;                 // two per TMEM lane quadrant, each takes every other block of 32 slots
constexpr int kGemmThreads = 96 + 32 * kEpiWarps;
constexpr int kSlotBlock = 16 * 32 * 2;      // 16 slots x 32 rows, f16: a tiled store
constexpr int kXchgBytes = 32 * 32 * 4;      // values on their way to the other warp of a team
// Results: gate/up one staging block per warp and an exchange buffer per team, down two staging blocks per warp.  Together
// with the ring little enough that the CTAs fit beside those of the sort and are set up when it ends.
constexpr size_t kGemmSmem = 1024 + kRingBytes + kEpiWarps * kSlotBlock + 4 * kXchgBytes;

// The sorted rows with a box for every number of slots that a CTA may hold (8, 16, ... 128): one copy per k-block.
struct SlotMaps {
  CUtensorMap m[kMaxBlockSlots / 16];
};
struct PairParams {
  const Block* table;
  const int* num_blocks;
  const float* wts;
  int mtiles, K, rows;  // rows: output rows of the projection
};

// Barriers between the two warps of a team (64 threads).
__device__ __forceinline__ void team_sync(int id) { asm volatile("barrier.cta.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ bool team_all(int id, bool v) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, 64, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
               : "=r"(r)
               : "r"((uint32_t)v), "r"(id)
               : "memory");
  return r != 0;
}

// One item = 256 weight rows x one block of slots, on a 2-CTA cluster.  CTA rank r holds 128 of the rows in its shared
// memory (gate/up: 64 gate rows and the 64 up rows that belong to them) and half of the block's slots per k-block, and the
// accumulators of its rows (TMEM lanes) x all slots (columns).  Roles and barriers as in gemm_pair_kernel (gemm.cu): warp 0
// loads weights, warp 2 slots, warp 1 of rank 0 issues the MMAs of both SMs, warps 3-10 store; two accumulators of 256
// columns.
// UP = true (gate/up): out = silu(gate) * up.  The gate values of a row are in lanes 0-63, the up values in lanes 64-127:
// the warp that holds the gate values of 32 rows and the one that holds the up values (a team) swap halves of 32 slots
// through shared memory and finish 16 slots each.  UP = false (down): out = value * routing weight.
// The down projection does not wait for the gate/up kernel before it fills its pipeline with weights: the block table is
// older, only the activations are new.
template <bool UP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
    moe_pair_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ SlotMaps tmX,
                         const __grid_constant__ CUtensorMap tmOut, const PairParams p, int* status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 2 * kEpiWarps);  // the epilogue warps of both CTAs
    }
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmOut);
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_s, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();  // the peer's barriers exist before anything is signalled on them
  cluster_wait();
  tc_fence_after();
  if (UP) {  // the next kernel on the stream may start its weights once everything before this one is complete
    grid_dependency_wait();
    grid_dependency_launch();
  } else {
    grid_dependency_launch();
  }
  const uint32_t tmem_base = tmem_base_s;
  volatile int* abort = &abort_s;
  const int items = __ldcg(p.num_blocks) * p.mtiles;
  const int stage_bytes = kABytes + __ldcg(p.num_blocks + 1) / 2 * 128;
  const int stages = min(kMaxStages, kRingBytes / stage_bytes);
  const int nk = (p.K + kBK - 1) / kBK;
  auto block_of = [&](int it) -> Block {
    const int4 v = it < items ? __ldcg(reinterpret_cast<const int4*>(p.table + it / p.mtiles)) : make_int4(0, 0, 16, 0);
    return {v.x, v.y, v.z, 0};
  };

  if (warp == 0 || warp == 2) {
    // ---- TMA producers (both CTAs): own weight rows (warp 0) and own half of the slots (warp 2), bytes counted on rank 0's
    // full barrier.  One copy per warp and k-block and little beside it: with both in one warp, six copies (boxes of 64
    // weight rows and 32 or 8 slots) and a division per k-block the issue took about 800 clocks per k-block and bound the
    // kernel whatever the operands' size.
    if (!UP && warp == 2) grid_dependency_wait();  // the activations
    const uint32_t bars = map_to_cta(&full[0], 0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int it = pair; ok && it < items; it += num_pairs) {
      const Block b = block_of(it);
      const int half = b.n / 2;
      const uint32_t bytes = 2 * (kABytes + half * 128);
      const int wrow = ((it % p.mtiles) * 2 + (int)rank) * (UP ? 64 : 128), xrow = b.row0 + (int)rank * half;
      const CUtensorMap* map = &tmX.m[b.n / 16 - 1];
      for (int kb = 0; kb < nk; ++kb) {
        ok = CTB_WARP_WAIT(&empty[stage], phase ^ 1, status, DEV_TIMEOUT_SLOT, abort);
        if (!ok) break;
        if (elect_one()) {
          unsigned char* dst = smem + stage * stage_bytes;
          if (warp == 0) {
            if (rank == 0) mbar_expect_tx(&full[stage], bytes);
            tma_load_4d_pair(dst, &tmW, kb * kBK, wrow, 0, b.expert, bars + stage * 8);
          } else {
            tma_load_3d_pair(dst + kABytes, map, kb * kBK, xrow, 0, bars + stage * 8);
          }
        }
        __syncwarp();
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ---- MMA issuer (rank 0 only): one instruction drives the tensor cores of both SMs
      int stage = 0, n = 0;
      uint32_t phase = 0;
      Block next = block_of(pair);
      for (int it = pair; it < items; it += num_pairs, ++n) {
        const uint32_t idesc = make_idesc(FMT_F16, 256, (uint32_t)next.n, 0, 0);
        next = block_of(it + num_pairs);
        const int acc = n & 1;
        const uint32_t acc_phase = (n >> 1) & 1;
        if (!CTB_WARP_WAIT(&acc_empty[acc], acc_phase ^ 1, status, DEV_TIMEOUT_SLOT, abort)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + acc * 256;
        bool ok = true;
        for (int kb = 0; kb < nk; ++kb) {
          ok = CTB_WARP_WAIT(&full[stage], phase, status, DEV_TIMEOUT_TMA, abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * stage_bytes), sb = sa + kABytes;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              mma_f16_ss_pair(d, make_sdesc_sw128(sa + k * 32, 0, 1024), make_sdesc_sw128(sb + k * 32, 0, 1024), idesc,
                              (kb | k) != 0);
            tc_commit_pair(&empty[stage], 3);
          }
          __syncwarp();
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        if (elect_one()) tc_commit_pair(&acc_full[acc], 3);
        __syncwarp();
      }
    }
  } else {
    // ---- epilogue: lane = output row (UP: gate or up row), 32 slots at a time -> this warp's staging block -> tiled stores
    const int sub = warp & 3, half = (warp - 3) >> 2;  // TMEM lanes [32 sub, 32 sub + 32), every other block of slots
    unsigned char* epi = smem + kRingBytes;
    __half* out = reinterpret_cast<__half*>(epi + (warp - 3) * (UP ? kSlotBlock : 2 * kSlotBlock));
    const int team = half * 2 + (sub & 1);
    const bool gate = sub < 2;
    // UP: [16 slots][32 lanes] to the up warp, then the same to the gate warp
    float* xchg = reinterpret_cast<float*>(epi + kEpiWarps * kSlotBlock + team * kXchgBytes) + lane;
    int n = 0;
    Block next = block_of(pair);
    for (int it = pair; it < items; it += num_pairs, ++n) {
      const Block b = next;
      next = block_of(it + num_pairs);
      const int acc = n & 1;
      bool ok = CTB_WARP_WAIT1(&acc_full[acc], (n >> 1) & 1, status, DEV_TIMEOUT_MMA, abort);
      if (UP) ok = team_all(1 + team, ok);  // both warps of a team go on or both stop
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * 256 + ((uint32_t)(sub * 32) << 16);
      const int m0 = UP ? (it % p.mtiles) * 128 + (int)rank * 64 + (sub & 1) * 32 : (it % p.mtiles) * 256 + (int)rank * 128 + sub * 32;
      uint32_t r[2][32];
      if (half * 32 < b.n) tmem_ld32(taddr + half * 32, r[0]);
#pragma unroll
      for (int i = 0; i < kMaxBlockSlots / 64; ++i) {
        const int c = i * 64 + half * 32;
        if (c >= b.n) break;  // uniform
        uint32_t(&v)[32] = r[i & 1];
        float4 w4[8];
        if constexpr (!UP) {  // routing weights of the 32 slots, the same for all lanes (row0 is a multiple of 16)
#pragma unroll
          for (int q = 0; q < 8; ++q)
            w4[q] = c + q * 4 < b.n ? __ldcg(reinterpret_cast<const float4*>(p.wts + b.row0 + c) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        tc_wait_ld();
        if (c + 64 < b.n) tmem_ld32(taddr + c + 64, r[(i + 1) & 1]);
        if constexpr (UP) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (gate) xchg[j * 32] = __uint_as_float(v[16 + j]);
            else xchg[(16 + j) * 32] = __uint_as_float(v[j]);
          }
          team_sync(1 + team);
          if (lane == 0) bulk_wait_read<0>();  // the previous store has read the staging block
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 16; ++j) {  // silu(g) * u with flush-to-zero and an approximate reciprocal (examples/moe.jl:117-124)
            const float got = xchg[(gate ? 16 + j : j) * 32];
            const float g = gate ? __uint_as_float(v[j]) : got, u = gate ? got : __uint_as_float(v[16 + j]);
            out[j * 32 + lane] = __float2half_rn(g * rcp_approx_ftz(1.0f + __expf(-g)) * u);
          }
        } else {
          if (lane == 0) bulk_wait_read<0>();  // the previous stores have read the staging blocks
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float4 w = w4[j / 4];
            const float wt = j % 4 == 0 ? w.x : j % 4 == 1 ? w.y : j % 4 == 2 ? w.z : w.w;
            out[j * 32 + lane] = __float2half_rn(__uint_as_float(v[j]) * wt);
          }
        }
        fence_proxy_async_smem();
        if (UP) team_sync(1 + team);  // the exchange buffer has been read
        else __syncwarp();
        if (lane == 0 && m0 < p.rows) {  // rows beyond the tensor are clipped, slots beyond the block are not stored
          if (UP) {
            const int first = c + (gate ? 0 : 16);
            if (first < b.n) tma_store_3d(&tmOut, out, m0, b.row0 + first, 0);
          } else {
            tma_store_3d(&tmOut, out, m0, b.row0 + c, 0);
            if (c + 16 < b.n) tma_store_3d(&tmOut, out + 16 * 32, m0, b.row0 + c + 16, 0);
          }
          bulk_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(&acc_empty[acc], 0));
    }
    bulk_wait<0>();  // this warp's stores are complete
  }
  // Neither CTA may leave (or free its TMEM) while the other can still read its shared memory, write its TMEM or
  // signal its barriers: every thread of both CTAs meets here, also after an abort.
  tc_fence_before();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
  if (!UP) grid_dependency_wait();  // a CTA without items must not let the next kernel overtake the one before this
}

// ------------------------------------------------------------------ combine
// out(:, t) = sum over the top-k slot outputs of token t, f16 like the reference's cache3 (examples/moe.jl:230,256), added
// in f32 in ascending slot order and rounded once.
__global__ void __launch_bounds__(256)
    moe_sorted_combine_kernel(const __half* __restrict__ slots, const int* __restrict__ pos_of, __half* __restrict__ out, int T,
                              int H, int topk) {
  grid_dependency_sync();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // over T*H/8
  const int h8 = H / 8;
  if (i >= (long long)T * h8) return;
  const int t = (int)(i / h8), h = (int)(i - (long long)t * h8) * 8;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  for (int s0 = 0; s0 < topk; s0 += 4) {
    uint4 v[4];
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (s0 + s < topk)
        v[s] = *reinterpret_cast<const uint4*>(slots + (long long)pos_of[(long long)t * topk + s0 + s] * H + h);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (s0 + s < topk) {
        const __half2* hv = reinterpret_cast<const __half2*>(&v[s]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __half22float2(hv[j]);
          acc[2 * j] += f.x;
          acc[2 * j + 1] += f.y;
        }
      }
    }
  }
  uint4 o;
  o.x = pack_f16x2(acc[0], acc[1]); o.y = pack_f16x2(acc[2], acc[3]);
  o.z = pack_f16x2(acc[4], acc[5]); o.w = pack_f16x2(acc[6], acc[7]);
  *reinterpret_cast<uint4*>(out + (long long)t * H + h) = o;
}

// ------------------------------------------------------------------ host side
struct Scratch {  // offsets in the context's scratch
  size_t xs, act, pos, wts, table, blocks, counts, bytes;
  int64_t rows;
  Scratch(int64_t T, int64_t H, int64_t I, int64_t E, int64_t topk) {
    auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
    const int64_t total = T * topk, used = std::min(total, E);  // experts with slots at most
    rows = (total + 15 * used + 15) & ~int64_t(15);
    xs = 0;  // sorted token rows; the down projection's results take their place
    act = xs + up((size_t)rows * H * 2);
    pos = act + up((size_t)rows * I * 2);
    wts = pos + up((size_t)total * 4);
    table = wts + up((size_t)rows * 4);
    blocks = table + up((size_t)(total / kMaxBlockSlots + used) * sizeof(Block));
    counts = blocks + 256;
    bytes = counts + (total > kSortLocal ? up((size_t)kSortCtas * (E + 1) * 4) : 0);
  }
};

template <bool UP>
int pair_clusters(ctb_ctx* ctx) {  // clusters of the kernel that the device runs at once (asked once per device)
  static int cached[16] = {0};
  int& c = cached[ctx->device & 15];
  if (c == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * ctx->sm_count);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = kGemmSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    cudaError_t e = cudaFuncSetAttribute(moe_pair_gemm_kernel<UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, moe_pair_gemm_kernel<UP>, &cfg);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
    }
    c = n;
  }
  return c;
}

template <bool UP>
int launch_projection(ctb_ctx* ctx, cudaStream_t st, const void* W, const void* X, void* out, int64_t K, int64_t wrows, int64_t N,
                      int64_t E, const Scratch& sc, unsigned char* ws, int64_t max_blocks) {
  CUtensorMap tw, to;
  SlotMaps tx;
  {
    // gate/up: a tile is 64 gate rows and the 64 up rows that belong to them; down: 128 rows
    uint64_t dims[4] = {(uint64_t)K, (uint64_t)N, UP ? 2u : 1u, (uint64_t)E};
    uint64_t str[3] = {(uint64_t)K * 2, (uint64_t)K * N * 2, (uint64_t)K * wrows * 2};
    uint32_t box[4] = {kBK, UP ? 64u : 128u, UP ? 2u : 1u, 1};
    int r = make_tmap(&tw, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, W, dims, str, box);
    if (r) return r;
  }
  for (int k = 0; k < kMaxBlockSlots / 16; ++k) {
    uint64_t dims[3] = {(uint64_t)K, (uint64_t)sc.rows, 1};
    uint64_t str[2] = {(uint64_t)K * 2, (uint64_t)K * sc.rows * 2};
    uint32_t box[3] = {kBK, 8u * (k + 1), 1};
    int r = make_tmap(&tx.m[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, X, dims, str, box);
    if (r) return r;
  }
  {
    uint64_t dims[3] = {(uint64_t)N, (uint64_t)sc.rows, 1};
    uint64_t str[2] = {(uint64_t)N * 2, (uint64_t)N * sc.rows * 2};
    uint32_t box[3] = {32, 16, 1};
    int r = make_tmap(&to, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, out, dims, str, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (r) return r;
  }
  PairParams p;
  p.table = reinterpret_cast<const Block*>(ws + sc.table);
  p.num_blocks = reinterpret_cast<const int*>(ws + sc.blocks);
  p.wts = reinterpret_cast<const float*>(ws + sc.wts);
  p.K = (int)K; p.rows = (int)N;
  p.mtiles = (int)((N + (UP ? 127 : 255)) / (UP ? 128 : 256));
  const int clusters = pair_clusters<UP>(ctx);
  if (clusters < 1) return fail(CTB_UNSUPPORTED, "ctb_moe_ffn: the device runs no CTA pairs");
  cudaError_t e = cudaFuncSetAttribute(moe_pair_gemm_kernel<UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
  if (e != cudaSuccess) return cuda_fail(e, "ctb_moe_ffn: shared memory opt-in");
  const int grid = 2 * (int)std::min<int64_t>(clusters, max_blocks * p.mtiles);
  e = launch_kernel(moe_pair_gemm_kernel<UP>, grid, kGemmThreads, kGemmSmem, st, 0, tw, tx, to, p, ctx->dev_status);
  if (e != cudaSuccess) return cuda_fail(e, "ctb_moe_ffn projection launch");
  return CTB_OK;
}

template <typename IdT>
int launch_sort(cudaStream_t st, const void* topk_ids, const SortParams& sp) {
  const IdT* ids = static_cast<const IdT*>(topk_ids);
  cudaError_t e = cudaSuccess;
  if (sp.counts)
    e = launch_kernel(moe_count_kernel<IdT>, kSortCtas, kSortThreads, 0, st, 0, ids, sp.T, sp.topk, sp.E, sp.total, sp.chunk,
                      const_cast<int*>(sp.counts));
  const size_t smem = (size_t)((3 + kSortWarps) * sp.E + 1) * sizeof(int);
  if (e == cudaSuccess) e = launch_kernel(moe_sort_gather_kernel<IdT>, kSortCtas, kSortThreads, smem, st, 0, ids, sp);
  return e == cudaSuccess ? (int)CTB_OK : cuda_fail(e, "ctb_moe_ffn sort launch");
}

}  // namespace

namespace ctb_internal {
size_t moe_ffn_workspace(int64_t T, int64_t H, int64_t I, int64_t E, int64_t topk) { return Scratch(T, H, I, E, topk).bytes; }
}  // namespace ctb_internal

extern "C" int ctb_moe_ffn(ctb_ctx* ctx, void* stream, const void* hidden, const void* w1, const void* w2,
                           const void* topk_weights, const void* topk_ids, int ids_bits, void* out, int64_t T, int64_t H,
                           int64_t I, int64_t E, int64_t topk, int tile_m, int tile_n, int tile_k) {
  CTB_CHECK_CTX(ctx);
  int r = moe_check_tile("ctb_moe_ffn", tile_m, tile_n, tile_k);
  if (r) return r;
  if (T <= 0 || H <= 0 || I <= 0 || E <= 0 || topk <= 0 || T * topk > (1 << 24))
    return fail(CTB_BAD_ARG, "ctb_moe_ffn: bad shape");
  if (E > kMaxExperts) return fail(CTB_UNSUPPORTED, "ctb_moe_ffn: at most %d experts", kMaxExperts);
  if (H % 8 || I % 8) return fail(CTB_BAD_ALIGN, "ctb_moe_ffn: hidden and intermediate sizes must be multiples of 8");
  if (ids_bits != 32 && ids_bits != 64) return fail(CTB_BAD_ARG, "ctb_moe_ffn: ids_bits must be 32 or 64");
  CTB_CHECK_DEV(hidden); CTB_CHECK_DEV(w1); CTB_CHECK_DEV(w2); CTB_CHECK_DEV(topk_weights); CTB_CHECK_DEV(topk_ids);
  CTB_CHECK_DEV(out);
  if ((uintptr_t)hidden % 16 || (uintptr_t)w1 % 16 || (uintptr_t)w2 % 16 || (uintptr_t)out % 16)
    return fail(CTB_BAD_ALIGN, "ctb_moe_ffn: 16-byte alignment of hidden, w1, w2");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const Scratch sc(T, H, I, E, topk);
  void* wsv;
  r = workspace(ctx, sc.bytes, &wsv, st);
  if (r) return r;
  unsigned char* ws = static_cast<unsigned char*>(wsv);
  const int total = (int)(T * topk);
  const int64_t max_blocks = total / kMaxBlockSlots + std::min<int64_t>(total, E);
  SortParams sp;
  sp.topk_w = static_cast<const __half*>(topk_weights);
  sp.X = static_cast<const uint4*>(hidden);
  sp.xs = reinterpret_cast<uint4*>(ws + sc.xs);
  sp.pos_of = reinterpret_cast<int*>(ws + sc.pos);
  sp.wts = reinterpret_cast<float*>(ws + sc.wts);
  sp.table = reinterpret_cast<Block*>(ws + sc.table);
  sp.num_blocks = reinterpret_cast<int*>(ws + sc.blocks);
  sp.counts = total > kSortLocal ? reinterpret_cast<int*>(ws + sc.counts) : nullptr;
  // With few slots the gate/up projection is bound by HBM, idle during the sort: fetch what its CTAs read first.
  sp.warm = total <= 2048 ? static_cast<const unsigned char*>(w1) : nullptr;
  sp.warm_expert = (long long)I * H * 2;
  sp.warm_tile = (int)(64 * H * 2);
  sp.warm_mtiles = (int)((I + 127) / 128);
  sp.T = (int)T; sp.topk = (int)topk; sp.E = (int)E; sp.vecs = (int)(H / 8); sp.total = total;
  sp.chunk = (total + kSortCtas - 1) / kSortCtas;
  sp.status = ctx->dev_status;
  r = ids_bits == 32 ? launch_sort<int>(st, topk_ids, sp) : launch_sort<long long>(st, topk_ids, sp);
  if (r) return r;
  // gate/up projection with the SwiGLU epilogue: act(:, row) = silu(Wg x) * (Wu x)
  r = launch_projection<true>(ctx, st, w1, ws + sc.xs, ws + sc.act, H, 2 * I, I, E, sc, ws, max_blocks);
  if (r) return r;
  // down projection scaled by the routing weight, one f16 row per slot (the reference's cache3)
  r = launch_projection<false>(ctx, st, w2, ws + sc.act, ws + sc.xs, I, H, H, E, sc, ws, max_blocks);
  if (r) return r;
  const long long n8 = T * (H / 8);
  cudaError_t e = launch_kernel(moe_sorted_combine_kernel, (unsigned)((n8 + 255) / 256), 256, 0, st, 0, (const __half*)(ws + sc.xs),
                                (const int*)(ws + sc.pos), (__half*)out, (int)T, (int)H, (int)topk);
  if (e != cudaSuccess) return cuda_fail(e, "ctb_moe_ffn combine launch");
  return CTB_OK;
}
