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
// whatever the block holds) 4096 tokens cost 25 % (50 % in pairs) of padding.  An expert with too many slots
// for one block (blocks_for) is cut into equal ones.
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "ctx.h"
#include "moe_place.h"
#include "ptx.cuh"

using namespace ctb;
using namespace ctb_internal;

namespace {

constexpr int kMaxExperts = 256;

// ------------------------------------------------------------------ sort and gather
constexpr int kSortThreads = 512, kSortCtas = 148;
constexpr int kSortThreadsEarly = 256;  // registers for a CTA of the gate/up kernel remain
constexpr int kSortLocal = 16384;  // up to this many slots every CTA counts all of them itself
// Up to this many slots the gate/up kernel starts beside the sort: it streams 28 MB of weights while the sort runs.  With more
// slots the weights bound it less than the rows, whose copies take 18 us instead of 6 beside that stream (8192 slots).
constexpr int kEarlySlots = 2048;

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
  int T, topk, E, vecs, total, chunk, early;
  int held;  // token rows that a CTA holds in shared memory; 0: they go through registers
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

// Adds every slot of expert e to tot[e] and, if `base` is given, those with a flat index below `lo` to base[e] (both in
// shared memory; SPLIT: to base[e] only); true if an id is out of range.  All threads of the CTA.
template <bool SPLIT, typename IdT>
__device__ __forceinline__ bool count_slots(const IdT* __restrict__ ids, int T, int topk, int E, int lo, int* tot, int* base) {
  bool bad = false;
  const int step = blockDim.x, total = T * topk;
  for (int m0 = threadIdx.x; m0 < total; m0 += 8 * step) {
    long long e[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) e[q] = m0 + q * step < total ? (long long)ids[m0 + q * step] - 1 : 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int m = m0 + q * step;
      if (m >= total) continue;
      if (e[q] < 0 || e[q] >= E) {
        bad = true;
        continue;
      }
      if (!SPLIT) atomicAdd(&tot[e[q]], 1);
      if (base) {
        const int slot = m / T;
        const bool before = (m - slot * T) * topk + slot < lo;
        if (SPLIT) atomicAdd(before ? &base[e[q]] : &tot[e[q]], 1);
        else if (before) atomicAdd(&base[e[q]], 1);
      }
    }
  }
  return bad;
}
// First row and first block of every expert from its number of slots (one warp; first[e] is added to).
__device__ __forceinline__ void scan_experts(bool ring, const int* tot, int E, int* first, int* bstart, int lane) {
  int rows = 0, blocks = 0;
  for (int e0 = 0; e0 < E; e0 += 32) {
    const int e = e0 + lane, c = e < E ? tot[e] : 0, padded = (c + 15) & ~15, nb = blocks_for(ring, c);
    int r = padded, b = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int rr = __shfl_up_sync(0xffffffffu, r, o), bb = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) { r += rr; b += bb; }
    }
    if (e < E) {
      first[e] += rows + r - padded;
      bstart[e] = blocks + b - nb;
    }
    rows += __shfl_sync(0xffffffffu, r, 31);
    blocks += __shfl_sync(0xffffffffu, b, 31);
  }
  if (lane == 0) bstart[E] = blocks;
}
// The blocks of expert e (c slots in nb blocks from row `row0` on); returns the slots of the largest.
__device__ __forceinline__ int write_blocks(Block* table, int e, int c, int nb, int row0) {
  const int size = ((c + nb - 1) / nb + 15) & ~15;
  for (int k = 0; k < nb; ++k) table[k] = {e, row0 + k * size, max((min(size, c - k * size) + 15) & ~15, 16), 0};
  return size;
}

// Ints of dynamic shared memory ahead of the rows (whole 128 bytes): slots per expert, those before the CTA's, the warps' counts,
// first blocks.
constexpr __host__ __device__ size_t sort_ints(int64_t E, int warps) { return (size_t)((3 + warps) * E + 1 + 31) & ~(size_t)31; }
constexpr size_t kHeldBytes = 160 * 1024;  // at most

// CTA c places the flat slots [c * chunk, (c + 1) * chunk) and copies their rows.  Nothing is exchanged between the CTAs:
// each counts all slots (or reads the chunks' counts) and so knows where every expert's rows and its own share of them
// start; the order inside an expert is the flat slot order, as in moe_align_tile_size (examples/moe.jl:142-183).
// Without the gate/up kernel beside it a CTA has room for the rows: each token's comes by one bulk copy while the slots are
// counted and leaves by one per choice, with nothing in registers (4096 tokens, top-2: through registers the kernel took
// 13.5 us, 5 of them for the rows once their places were known; now 9.5 and 2).
// A chain of latencies: 2.3 us to the counts, 4.3 to the table, then the rows.  The gate/up kernel does not wait for it: it
// is set up beside this one, counts the slots itself and streams weights meanwhile.
template <typename IdT, int kThreads>
__global__ void __launch_bounds__(kThreads) moe_sort_gather_kernel(const IdT* __restrict__ ids, const SortParams p) {
  constexpr int kWarps = kThreads / 32;
  constexpr bool HELD = kThreads == kSortThreads;  // without the gate/up kernel beside it
  extern __shared__ __align__(128) int sort_smem[];  // small where the next kernel's CTAs run beside this one's
  __shared__ int spos[kThreads];
  __shared__ int bad, nmax;
  __shared__ __align__(8) uint64_t rows_in;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, E = p.E, cta = blockIdx.x;
  int *tot = sort_smem, *base = tot + E, *wcount = base + E, *bstart = wcount + kWarps * E;  // [E], [E], [warps][E], [E + 1]
  for (int e = tid; e < E; e += kThreads) tot[e] = base[e] = 0;
  unsigned char* held = reinterpret_cast<unsigned char*>(sort_smem) + sort_ints(E, kWarps) * sizeof(int);  // [p.held] token rows
  const uint32_t row_bytes = (uint32_t)p.vecs * 16;
  if (tid == 0) {
    bad = nmax = 0;
    if (HELD) {
      mbar_init(&rows_in, 1);
      fence_mbar_init();
    }
  }
  __syncthreads();
  grid_dependency_wait();
  // the gate/up kernel reads the ids as well; if it waits for the table it is at least set up where a CTA of this kernel has ended
  grid_dependency_launch();
  const int lo = min(p.total, cta * p.chunk), hi = min(p.total, lo + p.chunk);
  // Which slots and rows are this CTA's is known from the start: the first are on their way before anything else is asked
  // for, ahead of the gate/up kernel's weights (behind them they took 5 us longer).
  uint4 v[8];
  auto load_rows = [&](int b0, int x0) {
    const int n = min(kThreads, hi - b0) * p.vecs;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int x = x0 + q * kThreads;
      if (x < n) {
        const int r = x / p.vecs;
        v[q] = __ldg(p.X + (long long)((b0 + r) / p.topk) * p.vecs + (x - r * p.vecs));
      }
    }
  };
  int e;
  __half weight;  // converted where it is used: nothing waits for it before the rows are requested
  auto load_slot = [&](int i) {
    e = -1;
    weight = __ushort_as_half(0);
    if (i < hi) {
      const int tok = i / p.topk, slot = i - tok * p.topk;
      e = (int)ids[(long long)slot * p.T + tok] - 1;
      weight = p.topk_w[(long long)slot * p.T + tok];
    }
  };
  // Slots at a time: their tokens are at most p.held.
  const int step = HELD && p.held ? min(kThreads, (p.held - 1) * p.topk) : kThreads;
  auto hold_rows = [&](int b0) {  // requests the rows of the tokens of the slots [b0, b0 + step)
    const int t0 = b0 / p.topk, n = (min(b0 + step, hi) - 1) / p.topk + 1 - t0;
    if (tid == 0) mbar_expect_tx(&rows_in, n * row_bytes);
    for (int r = tid; r < n; r += kThreads)
      bulk_g2s(held + (size_t)r * row_bytes, p.X + (long long)(t0 + r) * p.vecs, row_bytes, &rows_in);
  };
  if (HELD && p.held) {
    if (lo < hi) hold_rows(lo);
    load_slot(lo + tid);
  } else {
    load_slot(lo + tid);
    load_rows(lo, tid);
  }
  // ---- slots per expert: all of them, and those before this CTA's
  if (!p.counts) {
    if (count_slots<HELD>(ids, p.T, p.topk, E, lo, tot, base)) bad = 1;
  } else {
    for (int e = tid; e <= E; e += kThreads) {
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
    for (int i = lo + tid; i < hi; i += kThreads) p.pos_of[i] = 0;
    if (HELD && p.held && lo < hi) (void)mbar_wait(&rows_in, 0, p.status, DEV_TIMEOUT_TMA);
    return;
  }
  if (HELD && !p.counts) {
    for (int e = tid; e < E; e += kThreads) tot[e] += base[e];
    __syncthreads();
  }
  // ---- first row and first block of every expert
  if (warp == 0) scan_experts(HELD, tot, E, base, bstart, lane);
  __syncthreads();
  if (cta == 0) {  // the block table; this CTA has no slots before it: base is the experts' first row
    for (int e = tid; e < E; e += kThreads) {
      const int nb = bstart[e + 1] - bstart[e];
      if (nb) atomicMax(&nmax, write_blocks(p.table + bstart[e], e, tot[e], nb, base[e]));
    }
    __syncthreads();
    if (tid == 0) {
      p.num_blocks[0] = bstart[E];
      p.num_blocks[1] = nmax;
    }
    __syncthreads();
  }
  // ---- this CTA's slots, kThreads at a time: stable positions, then the rows
  int ebits = 1;
  while ((1 << ebits) < E) ++ebits;
  uint32_t phase = 0;
  for (int b0 = lo; b0 < hi; b0 += step) {
    if (HELD && p.held && b0 != lo) {
      bulk_wait_read<0>();  // the rows before these have left
      __syncthreads();
      hold_rows(b0);
    }
    for (int i = tid; i < kWarps * E; i += kThreads) wcount[i] = 0;
    __syncthreads();
    const int i = b0 + tid;
    if (b0 != lo) load_slot(i);
    if (HELD && tid >= step) e = -1;
    const unsigned grp = same_value(e, ebits);
    const int rank = __popc(grp & ((1u << lane) - 1));
    if (e >= 0 && rank == 0) wcount[warp * E + e] = __popc(grp);
    __syncthreads();
    if (tid < E) {
      int run = base[tid];
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
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
      p.wts[pos] = __half2float(weight);
    }
    if (HELD && p.held) {
      const bool ok = mbar_wait(&rows_in, phase, p.status, DEV_TIMEOUT_TMA);
      phase ^= 1;
      if (ok && e >= 0)
        bulk_s2g(p.xs + (long long)spos[tid] * p.vecs, held + (size_t)(i / p.topk - b0 / p.topk) * row_bytes, row_bytes);
      bulk_commit();
      if (__syncthreads_or(!ok)) {  // the copies must land before the CTA gives its shared memory back
        (void)mbar_wait(&rows_in, phase ^ 1, p.status, DEV_TIMEOUT_TMA);
        for (int j = b0 + step + tid; j < hi; j += kThreads) p.pos_of[j] = 0;  // the combine kernel finds valid positions
        break;
      }
      continue;
    }
    __syncthreads();
    const int n = min(kThreads, hi - b0) * p.vecs;
    for (int x0 = tid; x0 < n; x0 += 8 * kThreads) {
      if (b0 != lo || x0 != tid) load_rows(b0, x0);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int x = x0 + q * kThreads;
        if (x < n) {
          const int r = x / p.vecs;
          p.xs[(long long)spos[r] * p.vecs + (x - r * p.vecs)] = v[q];
        }
      }
    }
    __syncthreads();
  }
  if (HELD) bulk_wait_read<0>();  // this thread's rows have left shared memory
}

// ------------------------------------------------------------------ the two projections
constexpr int kBK = 64;                      // K elements per stage (128 bytes)
constexpr int kABytes = 128 * kBK * 2;       // a CTA's 128 weight rows of a k-block
constexpr int kMaxStages = 12;
constexpr int kRingBytes = 192 * 1024;
constexpr int kEpiWarps = 8;                 // two per TMEM lane quadrant, each takes every other block of 32 slots
constexpr int kGemmThreads = 96 + 32 * kEpiWarps;
constexpr int kTileBytes = 32 * 64 * 2;      // staged results: 32 slots x 64 rows, f16, 128-byte swizzle
// Warps that share a staging tile: gate/up the four quadrants (a CTA's 64 outputs), down two of them; two tiles each.
template <bool UP>
constexpr int kGroupThreads = UP ? 128 : 64;
template <bool UP>
constexpr size_t kGemmSmem = 1024 + kRingBytes + (size_t)(UP ? 2 : 4) * 2 * kTileBytes;
// The gate/up kernel's own block table behind it: slots, first rows and first blocks of E experts, then the blocks.
constexpr size_t own_table_bytes(int64_t E, int64_t blocks) { return (size_t)(((3 * E + 1) * 4 + 15) & ~15) + blocks * sizeof(Block); }
template <bool UP>
constexpr size_t kGemmSmemMost = kGemmSmem<UP> + (UP ? own_table_bytes(kMaxExperts, kEarlySlots / kMmaSlots + kMaxExperts) : 0);

// The sorted rows with a box for every number of slots that a CTA may hold (8, 16, ... 128): one copy per k-block.
struct SlotMaps {
  CUtensorMap m[kMmaSlots / 16];
};
struct PairParams {
  const Block* table;
  const int* num_blocks;
  const float* wts;
  int mtiles, K, rows;  // rows: output rows of the projection
  const void* ids;      // gate/up with at most kEarlySlots slots (not RING): the kernel builds its own table
  int ids_bits, T, topk, E;
};

// Barriers of `threads` threads (whole warps).
__device__ __forceinline__ void group_sync(int id, int threads) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ bool group_all(int id, int threads, bool v) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, %3, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
               : "=r"(r)
               : "r"((uint32_t)v), "r"(id), "r"(threads)
               : "memory");
  return r != 0;
}
// TMEM -> registers, 16 lanes x 32 columns: thread t holds, of the columns 8q + 2 (t mod 4) and the next, lane t / 4 in
// r[4q], r[4q + 1] and lane t / 4 + 8 in r[4q + 2], r[4q + 3].
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Four 8 x 8 matrices of 16-bit elements (register k of thread t: row t / 4, columns 2 (t mod 4) and the next of matrix k),
// stored transposed: lane l gives the address of column l mod 8 of matrix l / 8.
__device__ __forceinline__ void stmatrix4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

// One item = 256 weight rows x one block of slots, on a 2-CTA cluster.  CTA rank r holds 128 of the rows in its shared
// memory and half of the block's slots per k-block, and the accumulators of its rows (TMEM lanes) x all slots (columns).
// Roles and barriers as in gemm_pair_kernel (gemm.cu): warp 0 loads weights, warp 2 slots, warp 1 of rank 0 issues the MMAs
// of both SMs, warps 3-10 store; two accumulators of 256 columns.
// UP = true (gate/up): out = silu(gate) * up.  A CTA's rows are 64 gate and the 64 up rows that belong to them, in groups of
// eight in turn (a five-dimensional copy), so that a thread that reads two TMEM lanes eight apart has both values of an
// output.  UP = false (down): out = value * routing weight.  Results go through shared memory by transposing matrix stores
// (8 of 128 bytes per 32 slots and 16 outputs; element by element they were 48 of 64 bytes and shared the shared memory with
// the operands: with 4096 tokens the results cost 27 of 168 us that way, now 14 of 156).
// Neither projection waits for the kernel before it ahead of its first weights: the block table is older than it (down) or
// computed from the ids (gate/up); only the rows are new.
// The accumulators of an item follow those of the item before it in the ring of 512 columns: an item may begin when the one two
// before it has been read and, of the one before it, as many leading columns as it needs.  So a block can have more than 256
// slots and still start beside its predecessor's results.  With two halves of 256 columns an expert of 257 slots was two
// blocks, at the price of 256 slots each (a k-block of 144 slots took 330 ns, one of 256 slots 374): half of the experts at 4096
// tokens, top-2 over 32, where gate/up took 66 us and takes 57 now, down 39 and 35.  With at most kEarlySlots slots (not RING)
// large blocks are rare, and the two halves cost nothing in the roles' code (1 to 2 us of a step with few tokens).
// Up to 128 slots per block two k-blocks make a stage: the waits and issues of a stage take about 0.25 us, more than the weights
// of one k-block (100 tokens 86.3 -> 81.5 us, 1000 tokens 104.4 -> 102.6; larger blocks keep more and smaller stages in flight).
template <bool UP, bool RING>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
    moe_pair_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ SlotMaps tmX,
                         const __grid_constant__ CUtensorMap tmOut, const PairParams p, int* status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], part_empty[2][kParts];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s, nmax_s;
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
      for (int k = 0; RING && k < kParts; ++k) mbar_init(&part_empty[a][k], kEpiWarps);  // those of both that read block k
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
  if (!UP) grid_dependency_launch();
  const uint32_t tmem_base = tmem_base_s;
  volatile int* abort = &abort_s;
  const Block* table = p.table;
  int blocks, nmax;
  if (UP && !RING) {  // count the slots as the sort does
    int* tot = reinterpret_cast<int*>(smem_raw + kGemmSmem<UP>);
    int *first = tot + p.E, *bstart = first + p.E;
    Block* own = reinterpret_cast<Block*>(smem_raw + kGemmSmem<UP> + own_table_bytes(p.E, 0));
    for (int e = threadIdx.x; e < p.E; e += kGemmThreads) tot[e] = first[e] = 0;
    if (threadIdx.x == 0) nmax_s = 16;
    __syncthreads();
    const bool bad = p.ids_bits == 32 ? count_slots<false>(static_cast<const int*>(p.ids), p.T, p.topk, p.E, 0, tot, (int*)nullptr)
                                      : count_slots<false>(static_cast<const long long*>(p.ids), p.T, p.topk, p.E, 0, tot, (int*)nullptr);
    const bool none = __syncthreads_or(bad);
    if (warp == 0) scan_experts(RING, tot, p.E, first, bstart, lane);
    __syncthreads();
    for (int e = threadIdx.x; e < p.E; e += kGemmThreads) {
      const int nb = bstart[e + 1] - bstart[e];
      if (nb) atomicMax(&nmax_s, write_blocks(own + bstart[e], e, tot[e], nb, first[e]));
    }
    __syncthreads();
    table = own;
    blocks = none ? 0 : bstart[p.E];
    nmax = nmax_s;
  } else {
    if (UP) grid_dependency_wait();
    blocks = __ldcg(p.num_blocks);
    nmax = __ldcg(p.num_blocks + 1);
  }
  const int items = blocks * p.mtiles;
  const int per_stage = nmax <= 128 ? 2 : 1;  // k-blocks of a stage
  const int stage_bytes = per_stage * (kABytes + nmax / 2 * 128);
  const int stages = min(kMaxStages, kRingBytes / stage_bytes);
  const int nk = (p.K + kBK - 1) / kBK;
  auto block_of = [&](int it) -> Block {
    if (it >= items) return {0, 0, 16, 0};
    const Block* b = table + it / p.mtiles;
    return {b->expert, b->row0, b->n, 0};
  };

  if (warp == 0 || warp == 2) {
    // ---- TMA producers (both CTAs): own weight rows (warp 0) and own half of the slots (warp 2), bytes counted on rank 0's
    // full barrier.  One copy per warp and k-block and little beside it: with both in one warp, six copies (boxes of 64
    // weight rows and 32 or 8 slots) and a division per k-block the issue took about 800 clocks per k-block and bound the
    // kernel whatever the operands' size.
    if (warp == 2) {
      if (lane == 0) tma_prefetch_desc(&tmX.m[place<RING>(0, block_of(pair).n).first / 16 - 1]);
      grid_dependency_wait();  // the rows
      if (UP) grid_dependency_launch();  // the down projection may start its weights
    }
    const uint32_t bars = map_to_cta(&full[0], 0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int at = 0;
    Block next = block_of(pair);
    for (int it = pair; ok && it < items; it += num_pairs) {
      const Block b = RING ? next : block_of(it);
      if (RING) next = block_of(it + num_pairs);
      const Place pl = place<RING>(at, b.n);
      at = pl.next;
      const int half = b.n / 2, rest = b.n - pl.first;
      const uint32_t bytes = 2 * (kABytes + half * 128);
      const int wrow = ((it % p.mtiles) * 2 + (int)rank) * (UP ? 8 : 128), xrow = b.row0 + (int)rank * (pl.first / 2);
      const int xrest = b.row0 + pl.first + (int)rank * (rest / 2);
      const CUtensorMap *map = &tmX.m[pl.first / 16 - 1], *map_rest = &tmX.m[max(rest, 16) / 16 - 1];
      // fill(stage's memory, its barrier, first k, k-blocks) requests a stage
      auto walk = [&](auto fill) {
        for (int kb = 0; kb < nk; kb += per_stage) {
          ok = CTB_WARP_WAIT(&empty[stage], phase ^ 1, status, DEV_TIMEOUT_SLOT, abort);
          if (!ok) break;
          if (elect_one()) fill(smem + stage * stage_bytes, bars + stage * 8, kb * kBK, min(per_stage, nk - kb));
          __syncwarp();
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      };
      const int x_at = per_stage * kABytes, x_bytes = nmax / 2 * 128;
      if (warp == 0) {
        walk([&](unsigned char* dst, uint32_t bar, int k, int live) {
          if (rank == 0) mbar_expect_tx(&full[stage], live * bytes);
          for (int q = 0; q < live; ++q) {
            if (UP) tma_load_5d_pair(dst + q * kABytes, &tmW, k + q * kBK, 0, 0, wrow, b.expert, bar);
            else tma_load_3d_pair(dst + q * kABytes, &tmW, k + q * kBK, wrow, b.expert, bar);
          }
        });
      } else if (!RING || !rest) {
        walk([&](unsigned char* dst, uint32_t bar, int k, int live) {
          for (int q = 0; q < live; ++q) tma_load_3d_pair(dst + x_at + q * x_bytes, map, k + q * kBK, xrow, 0, bar);
        });
      } else {
        walk([&](unsigned char* dst, uint32_t bar, int k, int live) {
          for (int q = 0; q < live; ++q) {
            tma_load_3d_pair(dst + x_at + q * x_bytes, map, k + q * kBK, xrow, 0, bar);
            tma_load_3d_pair(dst + x_at + q * x_bytes + pl.first / 2 * 128, map_rest, k + q * kBK, xrest, 0, bar);
          }
        });
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ---- MMA issuer (rank 0 only): one instruction drives the tensor cores of both SMs
      int stage = 0, n = 0, at = 0, before = 0;  // before: columns of the item before this one
      uint32_t phase = 0;
      Block next = block_of(pair);
      for (int it = pair; it < items; it += num_pairs, ++n) {
        const Place pl = place<RING>(at, next.n);
        const int rest = next.n - pl.first, n32 = (next.n + 31) & ~31;
        const uint32_t idesc = make_idesc(FMT_F16, 256, (uint32_t)pl.first, 0, 0);
        const uint32_t idesc_rest = make_idesc(FMT_F16, 256, (uint32_t)max(rest, 16), 0, 0);
        const int shared = (before + pl.skipped + n32 - 512) / 32;  // leading blocks of the item before that this one overwrites
        at = pl.next;
        before = RING ? n32 : 0;
        next = block_of(it + num_pairs);
        const int acc = n & 1;
        const uint32_t acc_phase = (n >> 1) & 1;
        bool ok = CTB_WARP_WAIT(&acc_empty[acc], acc_phase ^ 1, status, DEV_TIMEOUT_SLOT, abort);
        for (int k = max(shared - 2, 0); ok && k < shared; ++k)  // the blocks go to two groups of warps in turn, in order
          ok = CTB_WARP_WAIT(&part_empty[acc ^ 1][k], ((n - 1) >> 1) & 1, status, DEV_TIMEOUT_SLOT, abort);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem_base + pl.col, d_rest = tmem_base + ((pl.col + pl.first) & 511);
        auto walk = [&](auto two_tag) {
          constexpr bool TWO = decltype(two_tag)::value;
          for (int kb = 0; kb < nk; kb += per_stage) {
            ok = CTB_WARP_WAIT(&full[stage], phase, status, DEV_TIMEOUT_TMA, abort);
            if (!ok) break;
            tc_fence_after();
            const int live = min(per_stage, nk - kb);
            const uint32_t sa0 = smem_u32(smem + stage * stage_bytes), sb0 = sa0 + per_stage * kABytes;
            if (elect_one()) {
              for (int q = 0; q < live; ++q) {
                const uint32_t sa = sa0 + q * kABytes, sb = sb0 + q * (nmax / 2 * 128);
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k)
                  mma_f16_ss_pair(d, make_sdesc_sw128(sa + k * 32, 0, 1024), make_sdesc_sw128(sb + k * 32, 0, 1024), idesc,
                                  (kb | q | k) != 0);
                if constexpr (TWO) {
                  const uint32_t sr = sb + pl.first / 2 * 128;
#pragma unroll
                  for (int k = 0; k < kBK / 16; ++k)
                    mma_f16_ss_pair(d_rest, make_sdesc_sw128(sa + k * 32, 0, 1024), make_sdesc_sw128(sr + k * 32, 0, 1024),
                                    idesc_rest, (kb | q | k) != 0);
                }
              }
              tc_commit_pair(&empty[stage], 3);
            }
            __syncwarp();
            if (++stage == stages) {
              stage = 0;
              phase ^= 1;
            }
          }
        };
        if constexpr (RING) {
          if (rest) walk(std::true_type());
          else walk(std::false_type());
        } else {
          walk(std::false_type());
        }
        if (!ok) break;
        if (elect_one()) tc_commit_pair(&acc_full[acc], 3);
        __syncwarp();
      }
    }
  } else {
    // ---- epilogue: 32 slots at a time -> staging tile [slot][64 outputs] of the group -> tiled store
    const int sub = warp & 3, half = (warp - 3) >> 2;  // TMEM lanes [32 sub, 32 sub + 32), every other block of slots
    const int group = UP ? half : half * 2 + (sub >> 1);
    const bool issuer = (UP ? sub == 3 : (sub & 1)) && lane == 0;
    const uint32_t tiles = smem_u32(smem + kRingBytes + group * 2 * kTileBytes);
    uint32_t flip = 0;  // the staging tile to fill next
    int n = 0, at = 0;
    Block next = block_of(pair);
    for (int it = pair; it < items; it += num_pairs, ++n) {
      const Block b = next;
      next = block_of(it + num_pairs);
      const int acc = n & 1;
      bool ok = CTB_WARP_WAIT1(&acc_full[acc], (n >> 1) & 1, status, DEV_TIMEOUT_MMA, abort);
      ok = group_all(1 + group, kGroupThreads<UP>, ok);  // the warps of a group go on or stop together
      if (!ok) break;
      tc_fence_after();
      const Place pl = place<RING>(at, b.n);
      at = pl.next;
      const uint32_t taddr = tmem_base + ((uint32_t)(sub * 32) << 16);
      const uint32_t acc_read = map_to_cta(&part_empty[acc][0], 0);
      const int m0 = UP ? (it % p.mtiles) * 128 + (int)rank * 64 : (it % p.mtiles) * 256 + (int)rank * 128 + (sub >> 1) * 64;
      uint32_t r[2][2][16];
      auto load = [&](int c, uint32_t (&v)[2][16]) {
        const uint32_t col = (pl.col + c) & 511;
        tmem_ld_16x32(taddr + col, v[0]);
        tmem_ld_16x32(taddr + (16u << 16) + col, v[1]);
      };
      if (half * 32 < b.n) load(half * 32, r[0]);
#pragma unroll
      for (int i = 0; i < (RING ? kMaxBlockSlots : kMmaSlots) / 64; ++i) {
        const int c = i * 64 + half * 32;
        if (c >= b.n) break;  // uniform
        uint32_t(&v)[2][16] = r[i & 1];
        float2 wt[4];
        if constexpr (!UP) {  // routing weights of this thread's slots
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int at = c + q * 8 + 2 * (lane & 3);
            wt[q] = at < b.n ? __ldcg(reinterpret_cast<const float2*>(p.wts + b.row0 + at)) : make_float2(0.f, 0.f);
          }
        }
        tc_wait_ld();
        if (RING && 2 * i + half < kParts) {  // this block of columns is in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(acc_read + (2 * i + half) * 8);
        }
        if (c + 64 < b.n) load(c + 64, r[(i + 1) & 1]);
        // lane l gives the address of slot c + l; 16-byte piece k of its 128 bytes lies at k ^ (l mod 8)
        const uint32_t row = tiles + flip * kTileBytes + lane * 128;
        auto piece = [&](int k) { return row + (uint32_t)((k ^ (lane & 7)) << 4); };
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t o[2][4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float a0 = __uint_as_float(v[h][4 * q]), a1 = __uint_as_float(v[h][4 * q + 1]);
            const float b0 = __uint_as_float(v[h][4 * q + 2]), b1 = __uint_as_float(v[h][4 * q + 3]);
            if constexpr (UP) {  // silu(g) * u with flush-to-zero and an approximate reciprocal (examples/moe.jl:117-124)
              o[0][q] = pack_f16x2(a0 * rcp_approx_ftz(1.0f + __expf(-a0)) * b0, a1 * rcp_approx_ftz(1.0f + __expf(-a1)) * b1);
            } else {
              o[0][q] = pack_f16x2(a0 * wt[q].x, a1 * wt[q].y);
              o[1][q] = pack_f16x2(b0 * wt[q].x, b1 * wt[q].y);
            }
          }
          if constexpr (UP) {
            stmatrix4_trans(piece(sub * 2 + h), o[0][0], o[0][1], o[0][2], o[0][3]);
          } else {
            stmatrix4_trans(piece((sub & 1) * 4 + h * 2), o[0][0], o[0][1], o[0][2], o[0][3]);
            stmatrix4_trans(piece((sub & 1) * 4 + h * 2 + 1), o[1][0], o[1][1], o[1][2], o[1][3]);
          }
        }
        fence_proxy_async_smem();
        if (issuer) bulk_wait_read<0>();  // the store before has read the other tile: free for everyone behind the barrier
        group_sync(1 + group, kGroupThreads<UP>);
        if (issuer && m0 < p.rows) {  // rows beyond the tensor are clipped, slots beyond the block are not stored
          const unsigned char* tile = smem + kRingBytes + (group * 2 + flip) * kTileBytes;
          tma_store_3d(&tmOut, tile, m0, b.row0 + c, 0);
          if (c + 16 < b.n) tma_store_3d(&tmOut, tile + kTileBytes / 2, m0, b.row0 + c + 16, 0);
          bulk_commit();
        }
        flip ^= 1;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        for (int k = half; RING && k < kParts; k += 2)  // blocks that this item does not have
          if (k * 32 >= b.n) mbar_arrive_cluster(acc_read + k * 8);
        mbar_arrive_cluster(map_to_cta(&acc_empty[acc], 0));
      }
    }
    bulk_wait<0>();  // this warp's stores are complete
  }
  // Neither CTA may leave (or free its TMEM) while the other can still read its shared memory, write its TMEM or
  // signal its barriers: every thread of both CTAs meets here, also after an abort.
  tc_fence_before();
  __syncthreads();
  let_copies_land(abort);
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
    blocks = table + up((size_t)(total / kMmaSlots + used) * sizeof(Block));
    counts = blocks + 256;
    bytes = counts + (total > kSortLocal ? up((size_t)kSortCtas * (E + 1) * 4) : 0);
  }
};

template <bool UP, bool RING>
int pair_clusters(ctb_ctx* ctx) {  // clusters of the kernel that the device runs at once (asked once per device)
  static int cached[16] = {0};
  int& c = cached[ctx->device & 15];
  if (c == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * ctx->sm_count);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = kGemmSmem<UP>;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    cudaError_t e = allow_smem(moe_pair_gemm_kernel<UP, RING>, kGemmSmemMost<UP>);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, moe_pair_gemm_kernel<UP, RING>, &cfg);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
    }
    c = n;
  }
  return c;
}

template <bool UP, bool RING>
int launch_projection(ctb_ctx* ctx, cudaStream_t st, const void* W, const void* X, void* out, int64_t K, int64_t wrows, int64_t N,
                      int64_t E, const Scratch& sc, unsigned char* ws, int64_t max_blocks, const void* ids, int ids_bits, int64_t T,
                      int64_t topk) {
  CUtensorMap tw, to;
  SlotMaps tx;
  if (UP) {  // 8 gate rows, the 8 up rows that belong to them, the next 8 gate rows, ...
    uint64_t dims[5] = {(uint64_t)K, 8, 2, (uint64_t)(N / 8), (uint64_t)E};
    uint64_t str[4] = {(uint64_t)K * 2, (uint64_t)K * N * 2, (uint64_t)K * 16, (uint64_t)K * wrows * 2};
    uint32_t box[5] = {kBK, 8, 2, 8, 1};
    int r = make_tmap(&tw, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, W, dims, str, box);
    if (r) return r;
  } else {
    uint64_t dims[3] = {(uint64_t)K, (uint64_t)wrows, (uint64_t)E};
    uint64_t str[2] = {(uint64_t)K * 2, (uint64_t)K * wrows * 2};
    uint32_t box[3] = {kBK, 128, 1};
    int r = make_tmap(&tw, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, W, dims, str, box);
    if (r) return r;
  }
  for (int k = 0; k < kMmaSlots / 16; ++k) {
    uint64_t dims[3] = {(uint64_t)K, (uint64_t)sc.rows, 1};
    uint64_t str[2] = {(uint64_t)K * 2, (uint64_t)K * sc.rows * 2};
    uint32_t box[3] = {kBK, 8u * (k + 1), 1};
    int r = make_tmap(&tx.m[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, X, dims, str, box);
    if (r) return r;
  }
  {
    uint64_t dims[3] = {(uint64_t)N, (uint64_t)sc.rows, 1};
    uint64_t str[2] = {(uint64_t)N * 2, (uint64_t)N * sc.rows * 2};
    uint32_t box[3] = {64, 16, 1};
    int r = make_tmap(&to, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, out, dims, str, box);
    if (r) return r;
  }
  PairParams p;
  p.table = reinterpret_cast<const Block*>(ws + sc.table);
  p.num_blocks = reinterpret_cast<const int*>(ws + sc.blocks);
  p.wts = reinterpret_cast<const float*>(ws + sc.wts);
  p.K = (int)K; p.rows = (int)N;
  p.mtiles = (int)((N + (UP ? 127 : 255)) / (UP ? 128 : 256));
  const int clusters = pair_clusters<UP, RING>(ctx);
  if (clusters < 1) return fail(CTB_UNSUPPORTED, "ctb_moe_ffn: the device runs no CTA pairs");
  p.ids = ids;
  p.ids_bits = ids_bits; p.T = (int)T; p.topk = (int)topk; p.E = (int)E;
  const size_t smem = kGemmSmem<UP> + (ids ? own_table_bytes(E, max_blocks) : 0);
  cudaError_t e = allow_smem(moe_pair_gemm_kernel<UP, RING>, kGemmSmemMost<UP>);
  if (e != cudaSuccess) return cuda_fail(e, "ctb_moe_ffn: shared memory opt-in");
  const int grid = 2 * (int)std::min<int64_t>(clusters, max_blocks * p.mtiles);
  e = launch_kernel(moe_pair_gemm_kernel<UP, RING>, grid, kGemmThreads, smem, st, 0, tw, tx, to, p, ctx->dev_status);
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
  auto kernel = sp.early ? moe_sort_gather_kernel<IdT, kSortThreadsEarly> : moe_sort_gather_kernel<IdT, kSortThreads>;
  const int threads = sp.early ? kSortThreadsEarly : kSortThreads;
  const size_t smem = sort_ints(sp.E, threads / 32) * sizeof(int) + (size_t)sp.held * sp.vecs * 16;
  // without the call the kernel's static shared memory counts against the same 48 KB
  if (e == cudaSuccess && !sp.early) e = allow_smem(kernel, sort_ints(kMaxExperts, threads / 32) * sizeof(int) + kHeldBytes);
  if (e == cudaSuccess) e = launch_kernel(kernel, kSortCtas, threads, smem, st, 0, ids, sp);
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
  const int64_t max_blocks = total / kMmaSlots + std::min<int64_t>(total, E);
  SortParams sp;
  sp.topk_w = static_cast<const __half*>(topk_weights);
  sp.X = static_cast<const uint4*>(hidden);
  sp.xs = reinterpret_cast<uint4*>(ws + sc.xs);
  sp.pos_of = reinterpret_cast<int*>(ws + sc.pos);
  sp.wts = reinterpret_cast<float*>(ws + sc.wts);
  sp.table = reinterpret_cast<Block*>(ws + sc.table);
  sp.num_blocks = reinterpret_cast<int*>(ws + sc.blocks);
  sp.counts = total > kSortLocal ? reinterpret_cast<int*>(ws + sc.counts) : nullptr;
  sp.early = total <= kEarlySlots;
  sp.T = (int)T; sp.topk = (int)topk; sp.E = (int)E; sp.vecs = (int)(H / 8); sp.total = total;
  sp.chunk = (total + kSortCtas - 1) / kSortCtas;
  // a chunk's tokens if they fit; two are needed for the slots to get on at all
  const int64_t tokens = (sp.chunk + topk - 1) / topk + 1, fit = (int64_t)kHeldBytes / (H * 2);
  sp.held = sp.early || fit < 2 ? 0 : (int)std::min(tokens, fit);
  sp.status = ctx->dev_status;
  r = ids_bits == 32 ? launch_sort<int>(st, topk_ids, sp) : launch_sort<long long>(st, topk_ids, sp);
  if (r) return r;
  auto project = [&](auto ring_tag) -> int {
    constexpr bool RING = decltype(ring_tag)::value;
    // gate/up projection with the SwiGLU epilogue: act(:, row) = silu(Wg x) * (Wu x)
    const int bad = launch_projection<true, RING>(ctx, st, w1, ws + sc.xs, ws + sc.act, H, 2 * I, I, E, sc, ws, max_blocks,
                                                  RING ? nullptr : topk_ids, ids_bits, T, topk);
    if (bad) return bad;
    // down projection scaled by the routing weight, one f16 row per slot (the reference's cache3)
    return launch_projection<false, RING>(ctx, st, w2, ws + sc.act, ws + sc.xs, I, H, H, E, sc, ws, max_blocks, nullptr, 0, T, topk);
  };
  r = sp.early ? project(std::false_type()) : project(std::true_type());
  if (r) return r;
  const long long n8 = T * (H / 8);
  cudaError_t e = launch_kernel(moe_sorted_combine_kernel, (unsigned)((n8 + 255) / 256), 256, 0, st, 0, (const __half*)(ws + sc.xs),
                                (const int*)(ws + sc.pos), (__half*)out, (int)T, (int)H, (int)topk);
  if (e != cudaSuccess) return cuda_fail(e, "ctb_moe_ffn combine launch");
  return CTB_OK;
}
