// Dense and batched GEMM for sm_100a: C(M,N[,b]) = A(M,K[,b]) * B(K,N[,b]),
// Julia column-major (counterparts of matmul_kernel, examples/matmul.jl:28-60,
// and batch_matmul_kernel, examples/batchmatmul.jl:15-56).
//
// f32 inputs run as TF32 tensor-core MMAs with f32 accumulation (the reference
// converts f32 -> tf32, examples/matmul.jl:49-52; the tensor core here reads the
// raw f32 bits from shared memory and ignores the low 13 mantissa bits, i.e.
// truncation instead of the reference's round-to-nearest-even); f16 inputs run
// as f16 MMAs with f32 accumulation and an f16 result.
//
// One persistent CTA per SM, 10 warps:
//   warp 0     TMA producer: per k-block, A as 128-byte-wide boxes (M contiguous,
//              "MN-major") and B as one box (K contiguous, "K-major"), 128B swizzle
//              (32-byte-atom flavour for the tf32 A operand),
//              into a ring of shared-memory stages guarded by mbarriers;
//   warp 1     MMA issuer: tcgen05.mma 128 x bn x (32 bytes of K) from shared-memory
//              descriptors into one of two 256-column TMEM accumulators;
//              tcgen05.commit frees the stage / publishes the accumulator;
//   warps 2-9  epilogue: tcgen05.ld the finished accumulator (lane = row m), stage
//              32 x 32 blocks in shared memory and store them by TMA while the MMA
//              warp already works on the next tile in the other accumulator.
// Tiles are bn columns wide, bn a multiple of 32 up to 256 (choose()).
// Out-of-range parts of edge tiles are zero-filled by TMA and clipped on store.
//
// Large problems run gemm_pair_kernel instead: the two CTAs of a 2-CTA cluster share one 256 x 256 tile
// (tcgen05 cta_group::2, the counterpart of the reference's num_ctas = 2 hint on this architecture,
// examples/matmul.jl:30).  Each CTA loads its own 128 rows of A and its own 128 columns of B per k-block, so an SM
// takes in 32 KB of operands per 128 x 256 x (128 bytes of K) of MMA work instead of 48 KB: operand delivery, not the
// tensor pipe, is what bounds the single-CTA kernel.  No load in this file is a cluster multicast.
#include <cuda_bf16.h>

#include <type_traits>

#include "ctx.h"
#include "ptx.cuh"

using namespace ctb;
using namespace ctb_internal;

namespace {

constexpr int kTileM = 128;
constexpr int kTileN = 256;
constexpr int kMaxStages = 8;
constexpr int kRingBytes = 192 * 1024;  // operand stages: as many of a tile's size as fit, at most kMaxStages
constexpr int kEpiWarps = 8;  // two per TMEM lane quadrant, each takes every other block of 32 columns
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kAccCols = kTileN;  // f32 accumulator columns per tile
constexpr uint32_t kTmemCols = 512;

// f32 accumulator -> result element (round to nearest even for the 16-bit types)
template <typename T>
__device__ __forceinline__ T from_f32(float v) {
  if constexpr (std::is_same<T, float>::value) return v;
  else if constexpr (std::is_same<T, __nv_bfloat16>::value) return __float2bfloat16_rn(v);
  else return __float2half_rn(v);
}

template <typename T>
struct Cfg {
  static constexpr int ES = sizeof(T);
  static constexpr int BK = 128 / ES;          // K elements per stage = one 128-byte swizzle span
  static constexpr int UK = 32 / ES;           // K per MMA instruction
  static constexpr int CHUNK_M = 128 / ES;     // M elements per A box (128 bytes)
  static constexpr int A_BOXES = kTileM / CHUNK_M;
  static constexpr int A_BOX_BYTES = BK * 128;  // BK rows of 128 bytes
  static constexpr int A_BYTES = A_BOXES * A_BOX_BYTES;
  static constexpr uint32_t FMT = sizeof(T) == 4 ? FMT_TF32 : std::is_same<T, __nv_bfloat16>::value ? FMT_BF16 : FMT_F16;
  // An MN-major tf32 operand must use the 128-byte swizzle with 32-byte atoms
  // (4 K-rows per swizzle period); 16-bit types use the ordinary 128-byte swizzle.
  static constexpr uint32_t A_LAYOUT = sizeof(T) == 4 ? SDESC_SW128_ATOM32 : SDESC_SW128;
  static constexpr uint32_t A_SBO = sizeof(T) == 4 ? 512 : 1024;
};

struct Params {
  int M, N, K, batch;
  long long ldc, strideC;
  int bn;  // columns of a tile: a multiple of 32, at most kTileN
  int stages, stage_bytes;  // per CTA; a stage is a multiple of 1024 bytes
  int tiles_m, tiles_n, num_tiles;
  // Results leave by tiled bulk stores (C starts on 16-byte boundaries) in blocks that end at or before this row.  A store
  // clips in units of 16 bytes: with M off that grid the last block would write into what lies behind C's columns.
  int tma_rows;
  // Split-K (single-CTA kernel, few tiles): a work unit is (tile, split); split s takes the k-blocks
  // [s * nk / splits, (s + 1) * nk / splits) and leaves its f32 accumulator tile in partial[unit], as blocks of
  // 32 columns x 32 rows (rows contiguous), four blocks per 32 columns; gemm_splitk_reduce_kernel adds the splits in
  // ascending order.
  int splits;
  float* partial;
};

// Results on their way out.  An epilogue warp owns 32 rows (lane = row) of 32 columns at a time: it writes them to a
// staging block in shared memory (a row of the block = 32 consecutive rows of a column of C, no bank conflicts)
// and lane 0 sends the block off with one tiled bulk store, which clips at the edges of C; the next block's TMEM load runs
// meanwhile.  Stored from registers, a tile of 128 x 256 cost about 10 us per CTA (12 x 1024 x 512 in bf16 with a single
// k-block: 23.5 us), more than its main loop for K up to 2000.  A warp has two blocks of 2 KB (16 columns in f32) and fills one
// while the other is read: with one, the last tile's results of 12 x 1000 x 515 x 776 in bf16 took 2.0 us and more.
constexpr int kStageBlock = 32 * 32 * 2;             // bytes of a staging block
constexpr int kEpiBytes = kEpiWarps * 2 * kStageBlock;
template <typename T>
constexpr int kStageCols = kStageBlock / (32 * (int)sizeof(T));
// One 32 x 32 block of a tile: r[j] = element (row m0 + lane, column n0 + j) of batch b.
template <typename T>
__device__ __forceinline__ void store_block(const Params& p, const void* tmapC, T* C, unsigned char* stage, int& sent,
                                            const uint32_t (&r)[32], int m0, int n0, int b, float* partial, int lane) {
  if (partial) {  // whole lines as they are: through the staging block a CTA with one unit waits for its last store
#pragma unroll
    for (int j = 0; j < 32; ++j) __stcg(partial + j * 32 + lane, __uint_as_float(r[j]));
  } else if (m0 + 32 <= p.tma_rows) {
#pragma unroll
    for (int h = 0; h < 32; h += kStageCols<T>) {
      unsigned char* block = stage + (sent++ & 1) * kStageBlock;
      if (lane == 0) bulk_wait_read<1>();  // the store before the previous one has read this block
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kStageCols<T>; ++j)
        reinterpret_cast<T*>(block)[j * 32 + lane] = from_f32<T>(__uint_as_float(r[h + j]));
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (m0 < p.M && n0 + h < p.N) tma_store_3d(tmapC, block, m0, n0 + h, b);
        bulk_commit();
      }
    }
  } else {
    const int m = m0 + lane;
    T* crow = C + (long long)b * p.strideC + m;
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (m < p.M && n0 + j < p.N) crow[(long long)(n0 + j) * p.ldc] = from_f32<T>(__uint_as_float(r[j]));
    __syncwarp();
  }
}

// A warp's share of a finished accumulator: every other block of 32 columns, the next one's TMEM load in flight while the
// current one is stored.
template <typename T>
__device__ __forceinline__ void store_tile(const Params& p, const void* tmapC, T* C, unsigned char* stage, int& sent,
                                           uint32_t taddr, int half, int m0, int n0, int b, float* partial, int lane) {
  const int nb = p.bn / 32;
  uint32_t r[2][32];
  if (half < nb) tmem_ld32(taddr + half * 32, r[0]);
#pragma unroll
  for (int i = 0; i < kTileN / 64; ++i) {
    const int c = 2 * i + half;
    if (c >= nb) break;  // uniform
    tc_wait_ld();
    if (c + 2 < nb) tmem_ld32(taddr + (c + 2) * 32, r[(i + 1) & 1]);
    store_block<T>(p, tmapC, C, stage, sent, r[i & 1], m0, n0 + c * 32, b, partial ? partial + c * 4096 : nullptr, lane);
  }
}

__device__ __forceinline__ void tile_coords(const Params& p, int t, int& b, int& tm, int& tn) {
  const int per_batch = p.tiles_m * p.tiles_n;
  b = t / per_batch;
  const int r = t - b * per_batch;
  // grouped order of examples/matmul.jl:13-24 (GROUP_SIZE_M = 8) for L2 reuse
  const int in_group = 8 * p.tiles_n;
  const int first = (r / in_group) * 8;
  const int gsz = min(p.tiles_m - first, 8);
  tm = first + (r % in_group) % gsz;
  tn = (r % in_group) / gsz;
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB,
                const __grid_constant__ CUtensorMap tmapC, T* __restrict__ C, const Params p, int* status) {
  using G = Cfg<T>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], kEpiWarps);
    }
    fence_mbar_init();
    tma_prefetch_desc(&tmapA);
    tma_prefetch_desc(&tmapB);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_dependency_sync();
  const uint32_t tmem_base = tmem_base_s;
  volatile int* abort = &abort_s;
  const int nk = (p.K + G::BK - 1) / G::BK;
  const int units = p.num_tiles * p.splits;

  if (warp == 0) {
    // ---- TMA producer: the whole warp walks the loop, one elected lane issues
    int stage = 0;
    uint32_t phase = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      int b, tm, tn;
      tile_coords(p, u / p.splits, b, tm, tn);
      const int sp = u % p.splits, kb_lo = sp * nk / p.splits, kb_hi = (sp + 1) * nk / p.splits;
      bool ok = true;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        ok = CTB_WARP_WAIT(&empty[stage], phase ^ 1, status, DEV_TIMEOUT_SLOT, abort);
        if (!ok) break;
        unsigned char* sa = smem + stage * p.stage_bytes;
        if (elect_one()) {
          mbar_expect_tx(&full[stage], G::A_BYTES + p.bn * 128);
#pragma unroll
          for (int j = 0; j < G::A_BOXES; ++j)
            tma_load_3d(sa + j * G::A_BOX_BYTES, &tmapA, tm * kTileM + j * G::CHUNK_M, kb * G::BK, b, &full[stage]);
          tma_load_3d(sa + G::A_BYTES, &tmapB, kb * G::BK, tn * p.bn, b, &full[stage]);
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the whole warp walks the loop, one elected lane issues
    const uint32_t idesc = make_idesc(G::FMT, kTileM, (uint32_t)p.bn, /*A MN-major*/ 1, /*B K-major*/ 0);
    int stage = 0;
    uint32_t phase = 0;
    int it = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++it) {
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      if (!CTB_WARP_WAIT(&acc_empty[acc], acc_phase ^ 1, status, DEV_TIMEOUT_SLOT, abort)) break;
      tc_fence_after();
      const uint32_t d = tmem_base + acc * kAccCols;
      const int sp = u % p.splits, kb_lo = sp * nk / p.splits, kb_hi = (sp + 1) * nk / p.splits;
      bool ok = true;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        ok = CTB_WARP_WAIT(&full[stage], phase, status, DEV_TIMEOUT_TMA, abort);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * p.stage_bytes);
        const uint32_t sb = sa + G::A_BYTES;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < G::BK / G::UK; ++k) {
            const uint64_t ad = make_sdesc(sa + k * G::UK * 128, G::A_BOX_BYTES, G::A_SBO, G::A_LAYOUT);
            const uint64_t bd = make_sdesc_sw128(sb + k * 32, 0, 1024);
            if constexpr (sizeof(T) == 4)
              mma_tf32_ss(d, ad, bd, idesc, ((kb - kb_lo) | k) != 0);
            else
              mma_f16_ss(d, ad, bd, idesc, ((kb - kb_lo) | k) != 0);
          }
          tc_commit(&empty[stage]);
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
      if (elect_one()) tc_commit(&acc_full[acc]);
      __syncwarp();
    }
  } else {
    const int sub = warp & 3;  // TMEM lanes [32*sub, 32*sub+32) belong to this warp
    const int half = (warp - 2) >> 2;
    unsigned char* epi = smem + kRingBytes + (warp - 2) * (2 * kStageBlock);
    int it = 0, sent = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++it) {
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      int b, tm, tn;
      tile_coords(p, u / p.splits, b, tm, tn);
      bool ok = CTB_WARP_WAIT(&acc_full[acc], acc_phase, status, DEV_TIMEOUT_MMA, abort);
      if (!ok) break;
      tc_fence_after();
      const int m0 = tm * kTileM + sub * 32;
      store_tile<T>(p, &tmapC, C, epi, sent, tmem_base + acc * kAccCols + ((uint32_t)(sub * 32) << 16), half, m0, tn * p.bn, b,
                    p.splits > 1 ? p.partial + (long long)u * (kTileM * kTileN) + sub * 1024 : nullptr, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
    }
    bulk_wait<0>();  // this warp's stores are complete
  }
  tc_fence_before();
  __syncthreads();
  let_copies_land(abort);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Adds the splits of every tile in ascending order and writes C.  A thread takes four consecutive rows of a column
// (16-byte loads; eight lanes cover a column's 32 rows of a block) and requests eight splits at a time.
template <typename T>
__global__ void __launch_bounds__(256)
    gemm_splitk_reduce_kernel(const float* __restrict__ partial, T* __restrict__ C, const Params p) {
  grid_dependency_sync();
  constexpr int kTileElems = kTileM * kTileN;
  const int per_tile = kTileM * p.bn / 4;
  const long long total = (long long)p.num_tiles * per_tile;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / per_tile), e = (int)(i - (long long)t * per_tile) * 4;
    const int block = e >> 10, col = (block >> 2) * 32 + ((e >> 5) & 31), row = (block & 3) * 32 + (e & 31);
    int b, tm, tn;
    tile_coords(p, t, b, tm, tn);
    const int m = tm * kTileM + row, n = tn * p.bn + col;
    if (m >= p.M || n >= p.N) continue;
    const float4* src = reinterpret_cast<const float4*>(partial + (long long)t * p.splits * kTileElems + e);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < p.splits; s0 += 8) {
      float4 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        v[q] = s0 + q < p.splits ? __ldcs(src + (long long)(s0 + q) * (kTileElems / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 8; ++q) {  // ascending split order
        acc.x += v[q].x;
        acc.y += v[q].y;
        acc.z += v[q].z;
        acc.w += v[q].w;
      }
    }
    T* dst = C + (long long)b * p.strideC + (long long)n * p.ldc + m;
    const float o[4] = {acc.x, acc.y, acc.z, acc.w};
    if (p.tma_rows && m + 3 < p.M) {  // C is aligned and m a multiple of four
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(dst) = acc;
      } else {
        T h[4] = {from_f32<T>(o[0]), from_f32<T>(o[1]), from_f32<T>(o[2]), from_f32<T>(o[3])};
        *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (m + q < p.M) dst[q] = from_f32<T>(o[q]);
    }
  }
}

// ---- CTA-pair kernel ---------------------------------------------------------------------------------------------
// Cluster of 2 CTAs = one 256 (M) x 256 (N) tile per step.  CTA rank r holds A rows [128 r, 128 r + 128) and
// B columns [128 r, 128 r + 128) of the tile in its shared memory and the accumulator rows [128 r, 128 r + 128) x 256
// columns in its TMEM.  Barriers: full[] lives in rank 0 and counts the bytes of both CTAs' loads; empty[] and
// acc_full[] exist in both CTAs and are arrived by rank 0's multicast commits; acc_empty[] lives in rank 0 and is
// arrived by the epilogue warps of both CTAs.
constexpr int kPairTileM = 256;

template <typename T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB,
                     const __grid_constant__ CUtensorMap tmapC, T* __restrict__ C, const Params p, int* status) {
  using G = Cfg<T>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
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
    tma_prefetch_desc(&tmapA);
    tma_prefetch_desc(&tmapB);
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_s, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();  // the peer's barriers exist before anything is signalled on them
  cluster_wait();
  tc_fence_after();
  grid_dependency_sync();
  const uint32_t tmem_base = tmem_base_s;
  volatile int* abort = &abort_s;
  const int nk = (p.K + G::BK - 1) / G::BK;

  if (warp == 0) {
    // ---- TMA producer (both CTAs): own halves of A and B, bytes counted on rank 0's full barrier
    int stage = 0;
    uint32_t phase = 0;
    for (int t = pair; t < p.num_tiles; t += num_pairs) {
      int b, tm, tn;
      tile_coords(p, t, b, tm, tn);
      const int m0 = tm * kPairTileM + (int)rank * kTileM, n0 = tn * p.bn + (int)rank * (p.bn / 2);
      bool ok = true;
      for (int kb = 0; kb < nk; ++kb) {
        ok = CTB_WARP_WAIT(&empty[stage], phase ^ 1, status, DEV_TIMEOUT_SLOT, abort);
        if (!ok) break;
        unsigned char* sa = smem + stage * p.stage_bytes;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * (G::A_BYTES + p.bn / 2 * 128));
          const uint32_t bar = map_to_cta(&full[stage], 0);
#pragma unroll
          for (int j = 0; j < G::A_BOXES; ++j)
            tma_load_3d_pair(sa + j * G::A_BOX_BYTES, &tmapA, m0 + j * G::CHUNK_M, kb * G::BK, b, bar);
          tma_load_3d_pair(sa + G::A_BYTES, &tmapB, kb * G::BK, n0, b, bar);
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ---- MMA issuer (rank 0 only): one instruction drives the tensor cores of both SMs
      const uint32_t idesc = make_idesc(G::FMT, kPairTileM, (uint32_t)p.bn, /*A MN-major*/ 1, /*B K-major*/ 0);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      for (int t = pair; t < p.num_tiles; t += num_pairs, ++it) {
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!CTB_WARP_WAIT(&acc_empty[acc], acc_phase ^ 1, status, DEV_TIMEOUT_SLOT, abort)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + acc * kAccCols;
        bool ok = true;
        for (int kb = 0; kb < nk; ++kb) {
          ok = CTB_WARP_WAIT(&full[stage], phase, status, DEV_TIMEOUT_TMA, abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * p.stage_bytes);
          const uint32_t sb = sa + G::A_BYTES;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < G::BK / G::UK; ++k) {
              const uint64_t ad = make_sdesc(sa + k * G::UK * 128, G::A_BOX_BYTES, G::A_SBO, G::A_LAYOUT);
              const uint64_t bd = make_sdesc_sw128(sb + k * 32, 0, 1024);
              if constexpr (sizeof(T) == 4)
                mma_tf32_ss_pair(d, ad, bd, idesc, (kb | k) != 0);
              else
                mma_f16_ss_pair(d, ad, bd, idesc, (kb | k) != 0);
            }
            tc_commit_pair(&empty[stage], 3);
          }
          __syncwarp();
          if (++stage == p.stages) {
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
    const int sub = warp & 3;  // TMEM lanes [32*sub, 32*sub+32) belong to this warp
    const int half = (warp - 2) >> 2;
    unsigned char* epi = smem + kRingBytes + (warp - 2) * (2 * kStageBlock);
    int it = 0, sent = 0;
    for (int t = pair; t < p.num_tiles; t += num_pairs, ++it) {
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      int b, tm, tn;
      tile_coords(p, t, b, tm, tn);
      bool ok = CTB_WARP_WAIT(&acc_full[acc], acc_phase, status, DEV_TIMEOUT_MMA, abort);
      if (!ok) break;
      tc_fence_after();
      const int m0 = tm * kPairTileM + (int)rank * kTileM + sub * 32;
      store_tile<T>(p, &tmapC, C, epi, sent, tmem_base + acc * kAccCols + ((uint32_t)(sub * 32) << 16), half, m0, tn * p.bn, b,
                    nullptr, lane);
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
  let_copies_land(abort);
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// How many 2-CTA clusters of gemm_pair_kernel the device runs at once (asked once per element type).
template <typename T>
int pair_clusters(ctb_ctx* ctx, size_t smem) {
  static int cached[16] = {0};  // per device; 0 = not asked yet, -1 = unavailable
  int& c = cached[ctx->device & 15];
  if (c == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * ctx->sm_count);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<T>, &cfg);
    c = (e == cudaSuccess && n > 0) ? n : -1;
    if (e != cudaSuccess) (void)cudaGetLastError();
  }
  return c;
}

// out[i] = in[i] rounded to TF32 precision, nearest even (NaNs stay NaNs): u + 0xFFF + bit 13, low 13 bits cleared.
__global__ void __launch_bounds__(256) tf32_round_kernel(const uint4* __restrict__ in, uint4* __restrict__ out, long long n4,
                                                         const uint32_t* __restrict__ in_tail, uint32_t* __restrict__ out_tail,
                                                         int tail) {
  grid_dependency_sync();
  auto rne = [](uint32_t u) {
    const bool nan = ((u >> 23) & 0xFFu) == 0xFFu && (u & 0x7FFFFFu) != 0;
    const uint32_t r = (u + 0xFFFu + ((u >> 13) & 1u)) & 0xFFFFE000u;
    return nan ? ((u & 0xFFFFE000u) | 0x2000u) : r;
  };
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    uint4 v = __ldcs(in + i);
    v.x = rne(v.x); v.y = rne(v.y); v.z = rne(v.z); v.w = rne(v.w);
    out[i] = v;
  }
  if (blockIdx.x == 0 && (int)threadIdx.x < tail) out_tail[threadIdx.x] = rne(in_tail[threadIdx.x]);
}

constexpr size_t kSmem = (size_t)kRingBytes + kEpiBytes + 1024;

// Kernel, tile width and number of splits of K, by an estimate of the clocks of the slowest CTA.  Per k-block (128 bytes of
// K) a tile of bn columns costs 2 bn clocks of tensor core per SM or, if that is more, the arrival of its operands (16 KB
// of A and bn or, in a pair, bn / 2 rows of 128 bytes of B, at about 55 bytes per clock and SM when all are loading: measured),
// and never less than the waits and issues of a stage (440); a tile's
// results need about 1000 + 4 bn clocks and hide behind the next tile's main loop, so a CTA pays per tile the larger of the two;
// filling the pipeline and the last tile's results come on top.  A split adds its partial tiles (written and read back
// through the L2) and a second kernel.  Narrow tiles fill the SMs and waste little of a ragged N, wide ones load less.
// Against the time of every choice on 90 products (f32, f16, bf16, 10 MFLOP to 137 GFLOP): the chosen one is 0.7 % from the
// best in the mean, 10 % at most; without the 440 it was 2.6 % and 21 %, narrow tiles being taken for long K (bf16
// 256 x 4096 x 4096: pairs of 64 columns 22.4 us, four splits of 256 columns 17.8).
struct Choice {
  bool pair;
  int bn, splits;
  int tile_m() const { return pair ? kPairTileM : kTileM; }
};
Choice choose(const ctb_ctx* ctx, long long M, long long N, long long nk, long long batch, int clusters) {
  Choice best = {false, kTileN, 1};
  double best_cost = 1e300;
  for (int pair = 0; pair <= (clusters > 0 && M > kTileM ? 1 : 0); ++pair)
    for (int bn = 32; bn <= kTileN; bn += 32) {
      if (bn > 32 && bn - 32 >= N) break;
      const long long tm = pair ? kPairTileM : kTileM;
      const long long tiles = ((M + tm - 1) / tm) * ((N + bn - 1) / bn) * batch, slots = pair ? clusters : ctx->sm_count;
      const double per_kb = std::max(std::max(440.0, 2.0 * bn), (16384.0 + (pair ? 64.0 : 128.0) * bn) / 55.0);
      for (int splits = 1; splits <= 16; ++splits) {
        if (splits > 1 && (pair || nk / splits < 4 || tiles * splits > slots)) break;
        const long long rounds = (tiles * splits + slots - 1) / slots;
        const double kloop = (double)((nk + splits - 1) / splits) * per_kb, epi = 1000.0 + 4.0 * bn;
        double cost = rounds * std::max(kloop, epi) + epi + 1500.0;
        if (splits > 1) cost += 6000.0 + (double)tiles * splits * kTileM * bn * 8.0 / slots / 60.0;
        if (cost < best_cost * 0.98) {
          best_cost = cost;
          best = {pair != 0, bn, splits};
        }
      }
    }
  return best;
}

template <typename T>
int launch(ctb_ctx* ctx, cudaStream_t st, const T* A, const T* B, T* C, int M, int N, int K, int batch, long long lda,
           long long ldb, long long ldc, long long sA, long long sB, long long sC) {
  using G = Cfg<T>;
  const CUtensorMapDataType dt = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                                          : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  size_t ws_used = 0;  // bytes of the context scratch taken by rounded operand copies (the split-K partials follow)
  if (sizeof(T) == 4 && ctx->tf32_rne) {
    // rounded copies with the layout of the originals (same leading dimensions and batch strides)
    // elements from the first to the last one that the arrays are known to hold
    const long long ea = (long long)(batch - 1) * sA + lda * (long long)(K - 1) + M;
    const long long eb = (long long)(batch - 1) * sB + ldb * (long long)(N - 1) + K;
    auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
    const size_t oa = 0, ob = up((size_t)ea * 4);
    ws_used = ob + up((size_t)eb * 4);
    const size_t partial_max = (size_t)ctx->sm_count * kTileM * kTileN * sizeof(float);  // split-K: at most one tile per SM
    void* ws = nullptr;
    int r = workspace(ctx, ws_used + partial_max, &ws, st);
    if (r) return r;
    float* A2 = reinterpret_cast<float*>(static_cast<unsigned char*>(ws) + oa);
    float* B2 = reinterpret_cast<float*>(static_cast<unsigned char*>(ws) + ob);
    const int rgrid = ctx->sm_count * 8;
    launch_kernel(tf32_round_kernel, rgrid, 256, 0, st, 0, reinterpret_cast<const uint4*>(A), reinterpret_cast<uint4*>(A2), ea / 4,
                                            reinterpret_cast<const uint32_t*>(A) + (ea & ~3ll),
                                            reinterpret_cast<uint32_t*>(A2) + (ea & ~3ll), (int)(ea & 3));
    launch_kernel(tf32_round_kernel, rgrid, 256, 0, st, 0, reinterpret_cast<const uint4*>(B), reinterpret_cast<uint4*>(B2), eb / 4,
                                            reinterpret_cast<const uint32_t*>(B) + (eb & ~3ll),
                                            reinterpret_cast<uint32_t*>(B2) + (eb & ~3ll), (int)(eb & 3));
    CTB_CHECK_LAUNCH("ctb_gemm operand rounding launch");
    A = reinterpret_cast<const T*>(A2);
    B = reinterpret_cast<const T*>(B2);
  }
  const int nk = (K + G::BK - 1) / G::BK;
  const Choice ch = choose(ctx, M, N, nk, batch, pair_clusters<T>(ctx, kSmem));
  CUtensorMap ta, tb, tc;
  {
    // A memory: [batch][K][M], M contiguous
    uint64_t dims[3] = {(uint64_t)M, (uint64_t)K, (uint64_t)batch};
    uint64_t str[2] = {(uint64_t)lda * G::ES, (uint64_t)(batch > 1 ? sA : lda * (long long)K) * G::ES};
    uint32_t box[3] = {(uint32_t)G::CHUNK_M, (uint32_t)G::BK, 1};
    int r = make_tmap(&ta, dt, 3, A, dims, str, box,
                      sizeof(T) == 4 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B);
    if (r) return r;
  }
  {
    // B memory: [batch][N][K], K contiguous; a CTA of a pair loads half of the tile's columns
    uint64_t dims[3] = {(uint64_t)K, (uint64_t)N, (uint64_t)batch};
    uint64_t str[2] = {(uint64_t)ldb * G::ES, (uint64_t)(batch > 1 ? sB : ldb * (long long)N) * G::ES};
    uint32_t box[3] = {(uint32_t)G::BK, (uint32_t)(ch.pair ? ch.bn / 2 : ch.bn), 1};
    int r = make_tmap(&tb, dt, 3, B, dims, str, box);
    if (r) return r;
  }
  Params p;
  p.M = M; p.N = N; p.K = K; p.batch = batch;
  p.ldc = ldc; p.strideC = sC;
  p.bn = ch.bn;
  p.stage_bytes = G::A_BYTES + (ch.pair ? ch.bn / 2 : ch.bn) * 128;
  p.stages = std::min(kMaxStages, kRingBytes / p.stage_bytes);
  p.tiles_m = (M + ch.tile_m() - 1) / ch.tile_m();
  p.tiles_n = (N + ch.bn - 1) / ch.bn;
  const long long nt = (long long)p.tiles_m * p.tiles_n * batch;
  if (nt * ch.splits > INT32_MAX) return fail(CTB_UNSUPPORTED, "ctb_gemm: too many tiles");
  p.num_tiles = (int)nt;
  p.splits = ch.splits;
  p.partial = nullptr;
  const bool c_aligned = (uintptr_t)C % 16 == 0 && ldc * G::ES % 16 == 0 && (batch == 1 || sC * G::ES % 16 == 0);
  p.tma_rows = !c_aligned ? 0 : (long long)M * G::ES % 16 == 0 ? INT32_MAX : M;
  tc = ta;  // not used when C is not aligned
  if (c_aligned) {
    uint64_t dims[3] = {(uint64_t)M, (uint64_t)N, (uint64_t)batch};
    uint64_t str[2] = {(uint64_t)ldc * G::ES, (uint64_t)(batch > 1 ? sC : ldc * (long long)N) * G::ES};
    uint32_t box[3] = {32, (uint32_t)kStageCols<T>, 1};
    int r = make_tmap(&tc, dt, 3, C, dims, str, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (r) return r;
  }
  if (ch.pair) {
    auto k = gemm_pair_kernel<T>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return cuda_fail(e, "ctb_gemm: shared memory opt-in");
    const int grid = 2 * (int)std::min<long long>(nt, pair_clusters<T>(ctx, kSmem));
    launch_kernel(k, grid, kThreads, kSmem, st, 0, ta, tb, tc, C, p, ctx->dev_status);
    CTB_CHECK_LAUNCH("ctb_gemm launch");
    return CTB_OK;
  }
  if (p.splits > 1) {
    void* ws = nullptr;
    int r = workspace(ctx, ws_used + (size_t)nt * p.splits * kTileM * kTileN * sizeof(float), &ws, st);
    if (r) return r;
    p.partial = reinterpret_cast<float*>(static_cast<unsigned char*>(ws) + ws_used);
  }
  auto k = gemm_kernel<T>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e != cudaSuccess) return cuda_fail(e, "ctb_gemm: shared memory opt-in");
  const int grid = (int)std::min<long long>(nt * p.splits, ctx->sm_count);
  launch_kernel(k, grid, kThreads, kSmem, st, 0, ta, tb, tc, C, p, ctx->dev_status);
  CTB_CHECK_LAUNCH("ctb_gemm launch");
  if (p.splits > 1) {
    const long long work = nt * kTileM * p.bn / 4;
    const int rgrid = (int)std::min<long long>((work + 255) / 256, (long long)ctx->sm_count * 8);
    launch_kernel(gemm_splitk_reduce_kernel<T>, rgrid, 256, 0, st, 0, p.partial, C, p);
    CTB_CHECK_LAUNCH("ctb_gemm split-K reduction launch");
  }
  return CTB_OK;
}

int gemm_common(ctb_ctx* ctx, void* stream, const void* A, const void* B, void* C, int64_t M, int64_t N, int64_t K,
                int64_t batch, int64_t lda, int64_t ldb, int64_t ldc, int64_t sA, int64_t sB, int64_t sC, int dtype,
                int tm, int tn, int tk, const char* who) {
  CTB_CHECK_CTX(ctx);
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0 || M > INT32_MAX || N > INT32_MAX || K > INT32_MAX || batch > 65535)
    return fail(CTB_BAD_ARG, "%s: bad shape M=%lld N=%lld K=%lld batch=%lld", who, (long long)M, (long long)N,
                (long long)K, (long long)batch);
  if (lda < M || ldb < K || ldc < M) return fail(CTB_BAD_ARG, "%s: leading dimension too small", who);
  if (!is_pow2(tm) || !is_pow2(tn) || !is_pow2(tk))
    return fail(CTB_UNSUPPORTED_TILE, "%s: tile sizes must be powers of two (got %d,%d,%d)", who, tm, tn, tk);
  if (dtype != CTB_F32 && dtype != CTB_F16 && dtype != CTB_BF16)
    return fail(CTB_BAD_ARG, "%s: dtype must be CTB_F32, CTB_F16 or CTB_BF16", who);
  CTB_CHECK_DEV(A); CTB_CHECK_DEV(B); CTB_CHECK_DEV(C);
  const int es = dtype == CTB_F32 ? 4 : 2;
  if ((lda * es) % 16 || (ldb * es) % 16 || (sA * es) % 16 || (sB * es) % 16 || (uintptr_t)A % 16 || (uintptr_t)B % 16)
    return fail(CTB_BAD_ALIGN, "%s: A and B need 16-byte aligned bases, leading dimensions and batch strides (TMA)", who);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == CTB_F32)
    return launch<float>(ctx, st, (const float*)A, (const float*)B, (float*)C, (int)M, (int)N, (int)K, (int)batch, lda,
                         ldb, ldc, sA, sB, sC);
  if (dtype == CTB_BF16)
    return launch<__nv_bfloat16>(ctx, st, (const __nv_bfloat16*)A, (const __nv_bfloat16*)B, (__nv_bfloat16*)C, (int)M, (int)N,
                                 (int)K, (int)batch, lda, ldb, ldc, sA, sB, sC);
  return launch<__half>(ctx, st, (const __half*)A, (const __half*)B, (__half*)C, (int)M, (int)N, (int)K, (int)batch,
                        lda, ldb, ldc, sA, sB, sC);
}

}  // namespace

extern "C" {

int ctb_gemm(ctb_ctx* ctx, void* stream, const void* A, const void* B, void* C, int64_t M, int64_t N, int64_t K,
             int64_t lda, int64_t ldb, int64_t ldc, int dtype, int tm, int tn, int tk) {
  return gemm_common(ctx, stream, A, B, C, M, N, K, 1, lda, ldb, ldc, 0, 0, 0, dtype, tm, tn, tk, "ctb_gemm");
}

int ctb_gemm_batched(ctb_ctx* ctx, void* stream, const void* A, const void* B, void* C, int64_t M, int64_t N,
                     int64_t K, int64_t batch, int64_t lda, int64_t ldb, int64_t ldc, int64_t strideA,
                     int64_t strideB, int64_t strideC, int dtype, int tm, int tn, int tk) {
  if (batch > 1 && (strideA < lda * K || strideB < ldb * N || strideC < ldc * N))
    return fail(CTB_BAD_ARG, "ctb_gemm_batched: batch strides overlap");
  return gemm_common(ctx, stream, A, B, C, M, N, K, batch, lda, ldb, ldc, strideA, strideB, strideC, dtype, tm, tn, tk,
                     "ctb_gemm_batched");
}

}  // extern "C"
