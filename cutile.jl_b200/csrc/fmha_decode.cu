// Flash attention forward for few query rows per key/value head (decode): all queries that share a key/value head - the
// heads of a group times the query positions, at most 16 rows - are one operand, and the keys are split over the GPU.
//
// What bounds it is HBM: K and V are read once, 256 bytes per key and key/value head, against a handful of rows.  The
// 128-row kernel (fmha.cu) spends a whole 128 x 128 tile on every query head, reads K and V once per query head and has
// one work item per head: 213 us for batch 32, 32 heads in 8 groups, 4000 keys (262 MB), against 40 us of traffic.
//
// Work is cut into blocks of 256 keys of one (batch, key/value head) pair.  The blocks of all pairs form one line that
// the CTAs (one per SM) share out in equal contiguous ranges, whatever the number of pairs and keys is: a CTA works
// through the end of one pair, whole pairs, the head of another, or through whole pairs only where that is as even.  With no more
// pairs than SMs the pairs are cut into as many equal parts as there are SMs for, and a CTA has a part of one pair only, unless too
// many SMs would be idle.  Inside a block each of the eight warps owns 32 keys: it has its own ring of stages that its lane 0 fills
// by TMA (K tile and V tile, 4 KB each, 128-byte swizzle, up to 192 KB in flight per SM), its own running maximum, sum and output,
// and waits for nobody until the CTA leaves the pair or comes to a cut.
// Cuts: probabilities are rounded to 16 bits relative to the warp's running maximum, and each running maximum is one that is exact,
// so a sum over fewer, longer pieces has the larger error (256 heads of 4000 keys in bf16: 2.18e-3 in whole pairs against 2.15e-3
// in ranges; 75 heads of 2000: 2.15e-3 and 2.08e-3).  CTAs that have whole pairs or equal parts therefore let their warps meet
// where a range would end as well, which costs them 0.2 to 1.7 us where there are such cuts (256 heads of 4000 keys 42.2 -> 42.6 us, in
// ranges 47.2; 75 heads of 2000 10.4 -> 11.8, in ranges 16.2), and the results of whole pairs are those of ranges bit for bit.
// S = Q K^T and O += P V are m16n8k16 tensor-core instructions on registers (a 128-row tcgen05 tile would be 88 % padding;
// the tensor work here is a few per cent of what either path delivers): Q stays in registers for the pair, K enters by
// ldmatrix, the probabilities go from the accumulator layout straight into the A operand, V by transposed ldmatrix.
// In the last block of a pair the warps behind the last key ask for nothing and have no part in what follows, and Q of the next
// pair is asked for before the warps meet: short heads are bound by these latencies (8192 heads of one row and 100 keys: 126 us
// when every warp took a tile and Q was asked for in its turn, 84 now; 3200 of 16 x 16: 70 and 39).
// Leaving a pair, the warps' results meet in shared memory; a pair that one CTA covers is written at once, otherwise the
// part goes to scratch and the CTA that arrives last adds the parts, each warp every eighth, in a fixed order (one thread per four
// outputs took them one after the other, with two divisions each: 32 heads over 4, 8000 keys 18.3 us, now 10.1).
#include <cuda_bf16.h>
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "ctx.h"
#include "ptx.cuh"

using namespace ctb;
using namespace ctb_internal;

namespace {

constexpr int kD = 64, kWarps = 8, kThreads = kWarps * 32, kTileKeys = 32, kBlockKeys = kWarps * kTileKeys;
constexpr int kTileBytes = kTileKeys * kD * 2;  // one K or V tile of a warp
constexpr int kPitch = kD + 4;                  // floats between rows of the warps' outputs in shared memory
constexpr int kMaxRows = 16;
constexpr int kPartFloats = kMaxRows * (kD + 2);
// Ends of ranges inside a pair or part, at most: with more pairs than SMs a range is no shorter than a pair (one end), with fewer
// no shorter than half of a part, rounded down (two).
constexpr int kMaxCuts = 2;

struct Params {
  const void* Q;
  void* Out;
  int seq_q, keys, seq_kv, group, rows;  // keys: up to the last one that some query sees
  int input_pos, causal, blocks_per_pair;
  long long blocks;
  int split;       // parts of a pair, a CTA each; 0: contiguous ranges of blocks; -1: contiguous ranges of whole pairs
  int cut_ranges;  // CUTS: the number of ranges
  float scale_log2;
  float* part;   // [CTA][first, last pair of its range][rows x (64 outputs), maxima, sums]
  unsigned* tickets;  // per CTA: parts left of the pair that begins in its range and ends in another's
};

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
template <bool BF16>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float lo, float hi) {
  if constexpr (BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    return pack_f16x2(lo, hi);
  }
}

// first block of CTA c, and the CTA that owns block b, when `blocks` are shared out over `grid` CTAs
__host__ __device__ __forceinline__ long long first_block(long long c, long long blocks, long long grid) {
  return c * blocks / grid;
}
__host__ __device__ __forceinline__ long long owner(long long b, long long blocks, long long grid) {
  return ((b + 1) * grid - 1) / blocks;
}

// R: query rows computed, 8 or 16 (the instructions have 16; the upper eight are zeros and skipped when R = 8).  CUTS: ends of
// ranges may lie inside what a CTA has of a pair (without the code for it short heads take 0.15 us less).
template <bool BF16, int R, bool CUTS>
__global__ void __launch_bounds__(kThreads, 1)
    fmha_decode_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const Params p,
                       int* status) {
  constexpr int kStages = R == 8 ? 3 : 2;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kWarps][kStages];
  __shared__ float ml[2][kWarps][kMaxRows];  // the warps' maxima and sums
  __shared__ int last_s;
  float* outs = reinterpret_cast<float*>(smem + kWarps * kStages * 2 * kTileBytes);  // [warp][R][kPitch]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (lane == 0) {
    for (int s = 0; s < kStages; ++s) mbar_init(&full[warp][s], 1);
    fence_mbar_init();
    if (warp == 0) {
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
    }
  }
  __syncwarp();
  grid_dependency_sync();

  const int cta = blockIdx.x, grid = gridDim.x;
  long long lo, hi;
  if (p.split < 0) {
    lo = first_block(cta, p.blocks / p.blocks_per_pair, grid) * p.blocks_per_pair;
    hi = first_block(cta + 1, p.blocks / p.blocks_per_pair, grid) * p.blocks_per_pair;
  } else if (p.split) {
    const int pr = cta / p.split, k = cta - pr * p.split;
    lo = (long long)pr * p.blocks_per_pair + k * p.blocks_per_pair / p.split;
    hi = (long long)pr * p.blocks_per_pair + (k + 1) * p.blocks_per_pair / p.split;
  } else {
    lo = first_block(cta, p.blocks, grid);
    hi = first_block(cta + 1, p.blocks, grid);
  }
  unsigned char* ring = smem + warp * (kStages * 2 * kTileBytes);
  // In the last block of a pair the keys end at some warp's tile; the warps behind it have none there.
  const int last_block = p.blocks_per_pair - 1, last_tiles = min(kWarps, (p.keys - last_block * kBlockKeys + kTileKeys - 1) / kTileKeys);
  auto tiles_of = [&](int block) { return block == last_block ? last_tiles : kWarps; };
  int issued = 0;
  // the block of the warp's next tile to ask for: pair, block of the pair, blocks left of the CTA's range
  int a_pair = (int)(lo / p.blocks_per_pair), a_block = (int)(lo - (long long)a_pair * p.blocks_per_pair), a_left = (int)(hi - lo);
  auto issue = [&]() {
    auto next = [&]() {
      --a_left;
      if (++a_block == p.blocks_per_pair) {
        a_block = 0;
        ++a_pair;
      }
    };
    while (a_left > 0 && warp >= tiles_of(a_block)) next();
    if (a_left <= 0) return;
    const int pair = a_pair, key0 = a_block * kBlockKeys + warp * kTileKeys, s = issued % kStages;
    next();
    if (lane == 0) {
      unsigned char* dst = ring + s * (2 * kTileBytes);
      mbar_expect_tx(&full[warp][s], 2 * kTileBytes);
      tma_load_3d(dst, &tmK, 0, key0, pair, &full[warp][s]);
      tma_load_3d(dst + kTileBytes, &tmV, 0, key0, pair, &full[warp][s]);
    }
    ++issued;
  };
  for (int s = 0; s < kStages; ++s) issue();

  // this lane's ldmatrix rows inside a tile: matrix lane / 8, row lane % 8
  const int mi = lane >> 3, mr = lane & 7;
  bool ok = true;
  int n = 0;  // tiles consumed
  // Q of a pair: rows g and g + 8 (row = head in group * seq_q + position)
  auto load_q = [&](uint32_t (&q)[4][4], int pair) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = g + 8 * h;
      const bool live = row < p.rows && (h == 0 || R == 16);
      const int head = row / p.seq_q, pos = row - head * p.seq_q;
      const uint32_t* src = reinterpret_cast<const uint32_t*>(
          static_cast<const uint16_t*>(p.Q) + (((long long)pair * p.group + head) * p.seq_q + pos) * kD);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        q[k][h] = live ? src[k * 8 + t] : 0u;
        q[k][2 + h] = live ? src[k * 8 + 4 + t] : 0u;
      }
    }
  };
  int lim[2];  // last visible key of the two rows
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = g + 8 * h, pos = row - row / p.seq_q * p.seq_q;
    lim[h] = p.causal ? min(p.input_pos + pos, p.seq_kv - 1) : p.seq_kv - 1;
  }
  float M_cut[kMaxCuts], L_cut[kMaxCuts];  // of the pair's pieces before the next cut
  float4 acc_cut[kMaxCuts];
  int cuts = 0;
  uint32_t q[4][4];
  uint32_t q_next[4][4];  // asked for before the warps of the last pair meet: with few keys a pair is over before its Q would have come
  load_q(q_next, (int)(lo / p.blocks_per_pair));
  // the next cut and the range of blocks that begins there (32 bits: see the launch)
  unsigned range = 0;
  long long cut = hi;
  auto next_cut = [&]() { cut = ++range * (unsigned)p.blocks / (unsigned)p.cut_ranges; };
  if constexpr (CUTS) {
    range = (((unsigned)lo + 1) * (unsigned)p.cut_ranges - 1) / (unsigned)p.blocks;  // that lo lies in
    next_cut();
  }
  int pair = (int)(lo / p.blocks_per_pair) - 1;
  for (long long b = lo; b < hi;) {
    if (!CUTS || cuts == 0) {
      ++pair;
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int h = 0; h < 4; ++h) q[k][h] = q_next[k][h];
    }
    const long long pair_first = (long long)pair * p.blocks_per_pair, pair_end = pair_first + p.blocks_per_pair;
    const long long end = CUTS ? min(min(hi, pair_end), cut) : min(hi, pair_end);
    int block = (int)(b - pair_first);
    const int live = tiles_of(block);  // warps that have keys of this part
    float o[8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
    // ---- the warp's tiles of the pair
    const long long mine_end = end == pair_end && warp >= last_tiles ? end - 1 : end;
    for (; b < mine_end; ++b, ++block) {
      const int s = n % kStages;
      if (ok) ok = CTB_WARP_WAIT(&full[warp][s], (n / kStages) & 1, status, DEV_TIMEOUT_TMA);
      if (!ok) continue;  // n stays at the tile that did not come
      ++n;
      const uint32_t sK = smem_u32(ring + s * (2 * kTileBytes)), sV = sK + kTileBytes;
      const int key0 = block * kBlockKeys + warp * kTileKeys;
      float sc[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // eight keys at a time
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[j][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {  // 32 of the 64 dimensions
          uint32_t r[4];
          ldmatrix4(r, sK + (j * 8 + mr) * 128 + (((kk * 4 + mi) ^ mr) << 4));
          mma16816<BF16>(sc[j], q[2 * kk], r[0], r[1]);
          mma16816<BF16>(sc[j], q[2 * kk + 1], r[2], r[3]);
        }
      }
      uint32_t pr[4][2];  // probabilities of eight keys, rows g and g + 8
#pragma unroll
      for (int h = 0; h < (R == 16 ? 2 : 1); ++h) {
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (key0 + j * 8 + 2 * t + e > lim[h]) sc[j][2 * h + e] = -INFINITY;
            mx = fmaxf(mx, sc[j][2 * h + e]);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float m_new = fmaxf(m[h], mx * p.scale_log2);
        const float ref = m_new == -INFINITY ? 0.f : m_new;
        const float alpha = ex2_approx_ftz(m[h] - ref);
        m[h] = m_new;
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p0 = ex2_approx_ftz(fmaf(sc[j][2 * h], p.scale_log2, -ref));
          const float p1 = ex2_approx_ftz(fmaf(sc[j][2 * h + 1], p.scale_log2, -ref));
          sum += p0 + p1;
          pr[j][h] = pack16<BF16>(p0, p1);
        }
        l[h] = l[h] * alpha + sum;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          o[j][2 * h] *= alpha;
          o[j][2 * h + 1] *= alpha;
        }
      }
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {  // 16 keys at a time
        const uint32_t a[4] = {pr[2 * kk][0], R == 16 ? pr[2 * kk][1] : 0u, pr[2 * kk + 1][0], R == 16 ? pr[2 * kk + 1][1] : 0u};
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // 16 dimensions
          uint32_t r[4];
          ldmatrix4_trans(r, sV + (kk * 16 + (mi & 1) * 8 + mr) * 128 + (((j * 2 + (mi >> 1)) ^ mr) << 4));
          mma16816<BF16>(o[2 * j], a, r[0], r[1]);
          mma16816<BF16>(o[2 * j + 1], a, r[2], r[3]);
        }
      }
      __syncwarp();  // every lane has read the stage
      issue();
    }
    b = end;
    if (CUTS ? end == pair_end && end < hi : pair_end < hi) load_q(q_next, pair + 1);
    // ---- leaving the pair: the warps' results meet
#pragma unroll
    for (int h = 0; h < (R == 16 ? 2 : 1); ++h) {
      if (warp >= live) break;
      l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
      l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
      if (t == 0) {
        ml[0][warp][g + 8 * h] = m[h];
        ml[1][warp][g + 8 * h] = l[h];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<float2*>(outs + (warp * R + g + 8 * h) * kPitch + j * 8 + 2 * t) = make_float2(o[j][2 * h], o[j][2 * h + 1]);
    }
    __syncthreads();
    const int row = tid >> 4, d0 = (tid & 15) * 4;  // 16 rows x 16 quarters of the outputs
    const bool mine = row < R && row < p.rows;
    float M = -INFINITY, L = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    auto meet = [&](auto all_tag) {  // the results of all warps, or of the first `live`
      constexpr bool ALL = decltype(all_tag)::value;
#pragma unroll
      for (int w = 0; w < kWarps; ++w)
        if (ALL || w < live) M = fmaxf(M, ml[0][w][row]);
      const float ref = M == -INFINITY ? 0.f : M;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {  // ascending: a fixed order
        if (!ALL && w >= live) break;
        const float f = ex2_approx_ftz(ml[0][w][row] - ref);
        const float4 v = *reinterpret_cast<const float4*>(outs + (w * R + row) * kPitch + d0);
        L += ml[1][w][row] * f;
        acc.x += v.x * f; acc.y += v.y * f; acc.z += v.z * f; acc.w += v.w * f;
      }
    };
    if (mine) {
      if (live == kWarps) meet(std::true_type());
      else meet(std::false_type());
    }
    if constexpr (CUTS) {
      if (end == cut && end < hi) next_cut();
      if (end < min(hi, pair_end)) {
#pragma unroll
        for (int k = 0; k < kMaxCuts; ++k)
          if (cuts == k) {
            M_cut[k] = M;
            L_cut[k] = L;
            acc_cut[k] = acc;
          }
        ++cuts;
        __syncthreads();  // the warps' results are overwritten by the next piece
        continue;
      }
      if (cuts) {  // the pieces in ascending order, as the parts of several CTAs below
        const float M_last = M, L_last = L;
        const float4 acc_last = acc;
#pragma unroll
        for (int k = 0; k < kMaxCuts; ++k)
          if (k < cuts) M = fmaxf(M, M_cut[k]);
        const float ref = M == -INFINITY ? 0.f : M;
        L = 0.f;
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
        auto add = [&](float m, float l, const float4& v) {
          const float f = ex2_approx_ftz(m - ref);
          L += l * f;
          acc.x += v.x * f; acc.y += v.y * f; acc.z += v.z * f; acc.w += v.w * f;
        };
#pragma unroll
        for (int k = 0; k < kMaxCuts; ++k)
          if (k < cuts) add(M_cut[k], L_cut[k], acc_cut[k]);
        add(M_last, L_last, acc_last);
        cuts = 0;
      }
    }
    auto write_out = [&]() {
      const float inv = rcp_approx_ftz(L);
      const int head = row / p.seq_q, pos = row - head * p.seq_q;
      uint2 v;
      v.x = pack16<BF16>(acc.x * inv, acc.y * inv);
      v.y = pack16<BF16>(acc.z * inv, acc.w * inv);
      *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p.Out) + (((long long)pair * p.group + head) * p.seq_q + pos) * kD + d0) = v;
    };
    if (lo <= pair_first && hi >= pair_end) {  // the whole pair was this CTA's
      if (mine) write_out();
      __syncthreads();  // the warps' results are overwritten by the next pair
      continue;
    }
    const int first_pair = (int)(lo / p.blocks_per_pair);
    float* part = p.part + ((long long)cta * 2 + (pair == first_pair ? 0 : 1)) * kPartFloats;
    if (mine) {
      *reinterpret_cast<float4*>(part + row * kD + d0) = acc;
      if (d0 == 0) {
        part[kMaxRows * kD + row] = M;
        part[kMaxRows * (kD + 1) + row] = L;
      }
    }
    const int c0 = p.split ? pair * p.split : (int)owner(pair_first, p.blocks, grid);
    const int c1 = p.split ? c0 + p.split - 1 : (int)owner(pair_end - 1, p.blocks, grid);
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      last_s = atomicInc(&p.tickets[c0], (unsigned)(c1 - c0)) == (unsigned)(c1 - c0);  // back to zero by the last
      __threadfence();
    }
    __syncthreads();
    if (last_s) {
      // warp w takes the parts c0 + w, c0 + w + 8, ...; a lane has two outputs of every row, lane r maximum and sum of row r
      const bool second = !p.split && first_block(c0, p.blocks, grid) != pair_first;  // c0's range begins before the pair
      auto part_of = [&](int c) { return p.part + ((long long)c * 2 + (c == c0 && second ? 1 : 0)) * kPartFloats; };
      const int r = lane & (R - 1);
      float mw = -INFINITY, lw = 0.f;
      float2 v[R];
#pragma unroll
      for (int k = 0; k < R; ++k) v[k] = make_float2(0.f, 0.f);
#pragma unroll 8
      for (int c = c0 + warp; c <= c1; c += kWarps) mw = fmaxf(mw, __ldcg(part_of(c) + kMaxRows * kD + r));
      const float ref = mw == -INFINITY ? 0.f : mw;
#pragma unroll 2
      for (int c = c0 + warp; c <= c1; c += kWarps) {
        const float* pc = part_of(c);
        float2 x[R];
#pragma unroll
        for (int k = 0; k < R; ++k) x[k] = __ldcg(reinterpret_cast<const float2*>(pc + k * kD) + lane);
        const float f = ex2_approx_ftz(__ldcg(pc + kMaxRows * kD + r) - ref);
        lw += __ldcg(pc + kMaxRows * (kD + 1) + r) * f;
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const float fk = __shfl_sync(0xffffffffu, f, k);
          if (k < p.rows) {
            v[k].x += x[k].x * fk;
            v[k].y += x[k].y * fk;
          }
        }
      }
      if (lane < R) {
        ml[0][warp][lane] = mw;
        ml[1][warp][lane] = lw;
      }
#pragma unroll
      for (int k = 0; k < R; ++k) *reinterpret_cast<float2*>(outs + (warp * R + k) * kPitch + 2 * lane) = v[k];
      __syncthreads();
      if (mine) {
        M = -INFINITY;
        L = 0.f;
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
        meet(std::true_type());
        write_out();
      }
    }
    __syncthreads();
  }
  if (!ok)  // a wait ran out: copies still in flight must land before the CTA gives its shared memory back
    for (int k = n; k < issued; ++k)
      (void)CTB_WARP_WAIT(&full[warp][k % kStages], (k / kStages) & 1, status, DEV_TIMEOUT_TMA);
}

}  // namespace

namespace ctb_internal {

bool fmha_decode_fits(int64_t seq_q, int group) { return seq_q * group <= kMaxRows; }

int fmha_decode(ctb_ctx* ctx, cudaStream_t st, const void* Q, const void* K, const void* V, void* Out, int64_t seq_q,
                int64_t seq_kv, int64_t heads, int64_t kv_heads, int64_t batch, float qk_scale, int input_pos, int64_t keys, bool causal,
                bool bf16, bool* taken) {
  const StreamScratch scratch(ctx, st);
  *taken = scratch.data != nullptr;
  if (!*taken) return CTB_OK;
  const CUtensorMapDataType tdt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tk, tv;
  const uint32_t box[3] = {kD, kTileKeys, 1};
  // The maps end at the last key that some query sees (see ctb_fmha_fwd); the copies fill with zeros there and read nothing.
  uint64_t dims[3] = {kD, (uint64_t)keys, (uint64_t)(kv_heads * batch)};
  uint64_t str[2] = {kD * 2, (uint64_t)seq_kv * kD * 2};
  int r = make_tmap(&tk, tdt, 3, K, dims, str, box);
  if (r) return r;
  r = make_tmap(&tv, tdt, 3, V, dims, str, box);
  if (r) return r;
  Params p;
  p.Q = Q; p.Out = Out;
  p.seq_q = (int)seq_q; p.keys = (int)keys; p.seq_kv = (int)seq_kv; p.group = (int)(heads / kv_heads);
  p.rows = p.group * p.seq_q;
  p.input_pos = input_pos; p.causal = causal ? 1 : 0;
  p.scale_log2 = qk_scale * 1.4426950408889634f;
  p.blocks_per_pair = (int)((keys + kBlockKeys - 1) / kBlockKeys);
  const int64_t pairs = kv_heads * batch;
  p.blocks = pairs * p.blocks_per_pair;
  int grid = (int)std::min<int64_t>(p.blocks, ctx->sm_count);
  const int ranges = grid;
  p.split = 0;
  if (pairs <= ctx->sm_count) {
    const int64_t split = std::min<int64_t>(p.blocks_per_pair, ctx->sm_count / pairs);
    const int64_t most = (p.blocks_per_pair + split - 1) / split;  // blocks of the largest part
    // A block (64 KB) takes an SM 1.46 us when all are loading and 0.93 by itself; ranges that cross from pair to pair cost 4.5 us
    // more, for the second pair that a CTA leaves.  One key/value head, 8192 keys: 29.2 us in ranges, 7.2 in parts; 120 heads of
    // 2000: 16.8 and 12.5; 75 heads of 6000, where one part each leaves half of the SMs idle, 25.2 and 26.3.
    const double parts = (double)most * std::max(0.93, 1.46 * (double)(split * pairs) / ctx->sm_count);
    if (parts <= 1.46 * (double)p.blocks / grid + 4.5) {
      p.split = (int)split;
      grid = (int)(split * pairs);
    }
  } else {
    // Whole pairs: HBM sets the pace while all are loading; at the end those with a pair more have it to themselves.
    // 256 heads of 4000 keys 45.9 us in ranges, 42.9 in whole pairs, 256 of 2000 26.9 and 23.4, 512 of 500 16.9 and 15.2;
    // 160 of 3000, where 12 CTAs have two pairs and 136 one, 25.0 and 29.0.
    const int64_t all = pairs / grid, more = pairs % grid;
    const double whole = p.blocks_per_pair * (1.46 * (double)all + (more ? std::max(0.93, 1.46 * (double)more / grid) : 0.));
    if (whole <= 1.46 * (double)p.blocks / grid + 4.5) p.split = -1;
  }
  // none where all ends of ranges are ends of pairs or parts
  p.cut_ranges = p.split && p.split != p.blocks_per_pair && p.blocks_per_pair > 1 && pairs % ranges ? ranges : 0;
  if (p.cut_ranges && p.blocks > UINT32_MAX / (ranges + 1)) {  // the kernel finds the cuts in 32 bits
    p.split = p.cut_ranges = 0;
    grid = ranges;
  }
  if ((size_t)grid * 2 * kPartFloats * sizeof(float) > kStreamScratchBytes || grid > kTickets)
    return fail(CTB_UNSUPPORTED, "ctb_fmha_fwd: more SMs than the split over keys has scratch for");
  p.part = scratch.data;
  p.tickets = scratch.tickets;
  const bool small = p.rows <= 8;
  const size_t smem = 1024 + (size_t)kWarps * (small ? 3 : 2) * 2 * kTileBytes + (size_t)kWarps * (small ? 8 : 16) * kPitch * 4;
  auto pick = [&](auto cuts) {
    constexpr bool CUTS = decltype(cuts)::value;
    return bf16 ? (small ? fmha_decode_kernel<true, 8, CUTS> : fmha_decode_kernel<true, 16, CUTS>)
                : (small ? fmha_decode_kernel<false, 8, CUTS> : fmha_decode_kernel<false, 16, CUTS>);
  };
  auto kern = p.cut_ranges ? pick(std::true_type()) : pick(std::false_type());
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "ctb_fmha_fwd: shared memory opt-in");
  launch_kernel(kern, grid, kThreads, smem, st, 0, tk, tv, p, ctx->dev_status);
  CTB_CHECK_LAUNCH("ctb_fmha_fwd launch");
  return CTB_OK;
}

}  // namespace ctb_internal
