// Row softmax for sm_100a.
//
// variant 0 ("single tile per row", the counterpart of softmax_tma_kernel,
//   examples/softmax.jl:18-42): persistent CTAs; each row is staged into shared
//   memory by one bulk async copy (cp.async.bulk + mbarrier) through a ring of
//   stages, normalised in registers, written back into the stage and stored
//   with a bulk copy shared->global, so loads and stores of neighbouring rows
//   overlap the arithmetic of the current one.
// variant 1 ("chunked", the counterpart of softmax_chunked_kernel, :48-100):
//   rows that fit the registers of a CTA and are 16-byte aligned take the
//   variant-0 kernel (one HBM read, one write; a chunk-by-chunk running
//   (max, sum) over bulk-copied chunks was measured 1.5x slower there because
//   it evaluates two exponentials per element).  Longer rows, of any alignment,
//   are kept whole in the shared memory of a cluster of CTAs: a running
//   (max, sum) over the chunks as they land, then a second pass that scales and
//   stores (still one HBM read, one write; for these rows the passes over
//   shared memory cost more than the second exponential).  Rows beyond that
//   (832 KB): a running (max, sum) per thread over chunks, re-read once.
// Both variants: rows of up to 1024 elements take a warp each.
//
// Both compute in f32 (examples/softmax.jl:32-35,92).  exp(x - max) is evaluated
// as ex2.approx((x - max)*log2(e)) (relative error about 2^-22 plus the rounding
// of the product) and the division as a multiplication by the exactly
// rounded reciprocal of the row sum, so that the kernel stays HBM-bound
// (2*M*N*sizeof(T) bytes per call) instead of instruction-bound.
#include <float.h>

#include <algorithm>

#include "ctx.h"
#include "ptx.cuh"

using namespace ctb;
using namespace ctb_internal;

namespace {

constexpr float kLog2e = 1.4426950408889634f;
// exp(x - m).  The subtraction comes first so that x == m gives exactly 1 and huge
// magnitudes cannot turn the rounding error of m*log2(e) into a wrong exponent.
__device__ __forceinline__ float exp_sub(float x, float m) { return ex2_approx_ftz((x - m) * kLog2e); }

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

struct __align__(8) Vec4h {
  __half2 a, b;
};

template <typename T>
struct Pack;  // 4 consecutive elements moved as one 16-byte (f32) or 8-byte (f16) access
template <>
struct Pack<float> {
  using type = float4;
  static __device__ __forceinline__ void unpack(const float4& v, float* f) {
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
  }
  static __device__ __forceinline__ float4 pack(const float* f) { return make_float4(f[0], f[1], f[2], f[3]); }
};
template <>
struct Pack<__half> {
  using type = Vec4h;
  static __device__ __forceinline__ void unpack(const Vec4h& v, float* f) {
    float2 x = __half22float2(v.a), y = __half22float2(v.b);
    f[0] = x.x; f[1] = x.y; f[2] = y.x; f[3] = y.y;
  }
  static __device__ __forceinline__ Vec4h pack(const float* f) {
    Vec4h v;
    v.a = __floats2half2_rn(f[0], f[1]);
    v.b = __floats2half2_rn(f[2], f[3]);
    return v;
  }
};

__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = red[0];
#pragma unroll
  for (int i = 1; i < kWarps; ++i) r = fmaxf(r, red[i]);
  __syncthreads();
  return r;
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = 0.f;
#pragma unroll
  for (int i = 0; i < kWarps; ++i) r += red[i];  // fixed order: deterministic
  __syncthreads();
  return r;
}

// ------------------------------------------------------------------ variant 0
// MAXV: packs of 4 elements kept in registers per thread (N <= 4*kThreads*MAXV).
template <typename T, int MAXV, int STAGES>
__global__ void __launch_bounds__(kThreads) softmax_staged_kernel(T* __restrict__ out, const T* __restrict__ in,
                                                                  int N, int M, long long ld_out, long long ld_in,
                                                                  int stage_bytes, int* status) {
  using P = typename Pack<T>::type;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[STAGES];
  __shared__ float red[kWarps];
  const int tid = threadIdx.x;
  const uint32_t row_bytes = (uint32_t)N * sizeof(T);
  const int npack = N / 4;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  grid_dependency_sync();

  const int first = blockIdx.x, step = gridDim.x;
  const int nrows = first < M ? (M - first + step - 1) / step : 0;

  // prologue: fill the ring
  if (tid == 0) {
    for (int i = 0; i < STAGES && i < nrows; ++i) {
      mbar_expect_tx(&full[i], row_bytes);
      bulk_g2s(smem + (size_t)i * stage_bytes, in + (long long)(first + i * step) * ld_in, row_bytes, &full[i]);
    }
  }

  bool alive = true;
  for (int i = 0; i < nrows && alive; ++i) {
    const int s = i % STAGES;
    const uint32_t parity = (i / STAGES) & 1;
    P* buf = reinterpret_cast<P*>(smem + (size_t)s * stage_bytes);
    if (!mbar_wait(&full[s], parity, status, DEV_TIMEOUT_TMA)) alive = false;
    alive = __syncthreads_and(alive);
    if (!alive) break;

    float x[MAXV][4];
    float mx = -FLT_MAX;
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      const int p = tid + v * kThreads;
      if (p < npack) {
        Pack<T>::unpack(buf[p], x[v]);
        mx = fmaxf(mx, fmaxf(fmaxf(x[v][0], x[v][1]), fmaxf(x[v][2], x[v][3])));
      }
    }
    mx = block_max(mx, red);
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      if (tid + v * kThreads < npack) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          x[v][k] = exp_sub(x[v][k], mx);
          s4[k] += x[v][k];
        }
      }
    }
    const float inv = 1.0f / block_sum((s4[0] + s4[1]) + (s4[2] + s4[3]), red);
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      const int p = tid + v * kThreads;
      if (p < npack) {
#pragma unroll
        for (int k = 0; k < 4; ++k) x[v][k] *= inv;
        buf[p] = Pack<T>::pack(x[v]);
      }
    }
    fence_proxy_async_smem();  // generic-proxy writes -> visible to the bulk store
    __syncthreads();
    if (tid == 0) {
      bulk_s2g(out + (long long)(first + i * step) * ld_out, buf, row_bytes);
      bulk_commit();
      // Refill the stage used by the PREVIOUS row: its store was committed one
      // iteration ago, so waiting for "all but the newest group" has read it.
      const int nxt = i - 1 + STAGES;
      if (i >= 1 && nxt < nrows) {
        bulk_wait_read<1>();
        const int ps = (i - 1) % STAGES;
        mbar_expect_tx(&full[ps], row_bytes);
        bulk_g2s(smem + (size_t)ps * stage_bytes, in + (long long)(first + nxt * step) * ld_in, row_bytes, &full[ps]);
      }
    }
  }
  if (tid == 0) bulk_wait<0>();  // stores complete before the CTA (and its smem) goes away
}

// ------------------------------------------------------------------ short rows
// Up to 1024 elements: one warp per row, the row in registers (element 32 i + lane, or 4 (32 i + lane) + k when VEC, the
// rows starting on vector boundaries), shuffles instead of barriers.  Bound by HBM for many rows (8192 x 1000 f32: a CTA
// per row through a ring of stages spends its time on two block reductions per 4 KB), by one load latency for few.
template <typename T, int NE, bool VEC>  // NE: elements per lane
__global__ void __launch_bounds__(128) softmax_warp_kernel(T* __restrict__ out, const T* __restrict__ in, int N, int M,
                                                           long long ld_out, long long ld_in) {
  grid_dependency_sync();
  const int lane = threadIdx.x & 31;
  for (int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < M; row += gridDim.x * (blockDim.x >> 5)) {
    const T* src = in + (long long)row * ld_in;
    T* dst = out + (long long)row * ld_out;
    float x[NE];
    if constexpr (VEC) {
#pragma unroll
      for (int i = 0; i < NE / 4; ++i) {
        const int p = i * 32 + lane;
        if (p * 4 < N) {
          Pack<T>::unpack(reinterpret_cast<const typename Pack<T>::type*>(src)[p], &x[4 * i]);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) x[4 * i + k] = -INFINITY;
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < NE; ++i) x[i] = i * 32 + lane < N ? (float)src[i * 32 + lane] : -INFINITY;
    }
    float mx = -FLT_MAX;
#pragma unroll
    for (int i = 0; i < NE; ++i) mx = fmaxf(mx, x[i]);
    mx = warp_max(mx);
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < NE; ++i) {
      x[i] = exp_sub(x[i], mx);  // 0 beyond the row
      s4[i & 3] += x[i];
    }
    const float inv = 1.0f / warp_sum((s4[0] + s4[1]) + (s4[2] + s4[3]));
#pragma unroll
    for (int i = 0; i < NE; ++i) x[i] *= inv;
    if constexpr (VEC) {
#pragma unroll
      for (int i = 0; i < NE / 4; ++i)
        if ((i * 32 + lane) * 4 < N) reinterpret_cast<typename Pack<T>::type*>(dst)[i * 32 + lane] = Pack<T>::pack(&x[4 * i]);
    } else {
#pragma unroll
      for (int i = 0; i < NE; ++i)
        if (i * 32 + lane < N) dst[i * 32 + lane] = (T)x[i];
    }
  }
}

// Up to 8192 elements in rows that do not start on vector boundaries: one CTA per row, the row in registers, element by
// element (a warp still covers whole lines), all of a thread's loads in flight at once.
template <typename T, int NE>
__global__ void __launch_bounds__(kThreads) softmax_regs_kernel(T* __restrict__ out, const T* __restrict__ in, int N, int M,
                                                                long long ld_out, long long ld_in) {
  __shared__ float red[kWarps];
  grid_dependency_sync();
  const int tid = threadIdx.x;
  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    const T* src = in + (long long)row * ld_in;
    T* dst = out + (long long)row * ld_out;
    float x[NE];
    float mx = -FLT_MAX;
#pragma unroll
    for (int i = 0; i < NE; ++i) x[i] = i * kThreads + tid < N ? (float)src[i * kThreads + tid] : -INFINITY;
#pragma unroll
    for (int i = 0; i < NE; ++i) mx = fmaxf(mx, x[i]);
    mx = block_max(mx, red);
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < NE; ++i) {
      x[i] = exp_sub(x[i], mx);
      s4[i & 3] += x[i];
    }
    const float inv = 1.0f / block_sum((s4[0] + s4[1]) + (s4[2] + s4[3]), red);
#pragma unroll
    for (int i = 0; i < NE; ++i)
      if (i * kThreads + tid < N) dst[i * kThreads + tid] = (T)(x[i] * inv);
  }
}

// ------------------------------------------------------------------ variant 1, long rows of any alignment
// Rows too long for the registers of a CTA: a cluster of C CTAs keeps the whole row in its shared memory, so HBM is
// read once and written once.  C is the smallest power of two with at most 104 KB per CTA, so that two or more CTAs share
// an SM and one loads while another computes or stores (one CTA per SM that held a whole row: 5400 GB/s on 1024 x 32768).
// The 16-byte aligned middle of the row arrives in chunks of kChunkVecs vectors, one bulk copy and mbarrier each; up to
// one vector's elements before and after it are loaded one by one by rank 0, so rows may start anywhere (1024 x 50001 f32:
// 227 us with scalar loads and a second read).  One online pass takes the running maximum and sum of exponentials of each
// chunk as it lands, the CTAs send them to each other (asynchronous stores that count on an mbarrier of the receiver, two sets of
// slots; with a cluster barrier per row, whose release waits for the stores of the row before, 1024 x 50001 f32 took 76.3 us, now
// 73.4, 800 x 65000 f16 51.3 and 44.9), and a second pass evaluates the exponentials again, scales and stores; a chunk's part of the buffer takes the
// next row's chunk as soon as it was read.
constexpr int kRowThreads = 512;
constexpr int kChunkVecs = 1024;
constexpr int kMaxChunks = 7;
constexpr int kMaxCluster = 8;
constexpr size_t kLongBytes = 104 * 1024;  // of a row, per CTA
template <typename T>
__device__ __forceinline__ void unpack16(const uint4& q, float (&f)[16 / sizeof(T)]) {
  if constexpr (sizeof(T) == 4) {
    f[0] = __uint_as_float(q.x); f[1] = __uint_as_float(q.y); f[2] = __uint_as_float(q.z); f[3] = __uint_as_float(q.w);
  } else {
    const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = __half22float2(h[i]);
      f[2 * i] = v.x;
      f[2 * i + 1] = v.y;
    }
  }
}
template <typename T>
__global__ void __launch_bounds__(kRowThreads) softmax_long_kernel(T* __restrict__ out, const T* __restrict__ in, int N, int M,
                                                                   long long ld_out, long long ld_in, int per, int C,
                                                                   int* status) {
  constexpr int V = 16 / (int)sizeof(T);
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[kMaxChunks];
  // Maximum and sum of every warp, for even and odd rows.  Read one by one: as vectors they bring the f32 kernel to 37 registers,
  // three CTAs per SM instead of four (700 x 8200 12.3 us instead of 11.4, 300 x 27001 17.4 and 14.8).
  __shared__ float red[2][2][kRowThreads / 32];
  __shared__ __align__(8) float2 peers[2][kMaxCluster];         // and of every CTA of the cluster
  __shared__ __align__(8) uint64_t met[2];               // all of peers[] have come
  __shared__ volatile int given_up;                      // they have not: no further arrival, message or wait
  const int tid = threadIdx.x;
  const int rank = C > 1 ? (int)cluster_ctarank() : 0, team = blockIdx.x / C, teams = gridDim.x / C;
  if (tid == 0) {
    for (int c = 0; c < kMaxChunks; ++c) mbar_init(&full[c], 1);
    mbar_init(&met[0], 1);
    mbar_init(&met[1], 1);
    given_up = 0;
    fence_mbar_init();
  }
  __syncthreads();
  if (C > 1) {  // the peers' shared memory and barriers exist
    cluster_arrive();
    cluster_wait();
  }
  grid_dependency_sync();
  uint4* buf = reinterpret_cast<uint4*>(smem);
  // the row's elements before the first 16-byte boundary, and the vectors [v0, v1) of the middle that are this CTA's
  auto layout = [&](int row, const T*& src, int& head, int& nvec, int& v0, int& v1) {
    src = in + (long long)row * ld_in;
    head = min(N, (int)((16 - ((uintptr_t)src & 15)) & 15) / (int)sizeof(T));
    nvec = (N - head) / V;
    v0 = min(nvec, rank * per);
    v1 = min(nvec, v0 + per);
  };
  uint32_t pending = 0;  // thread 0: chunks whose copy is under way
  auto load_chunk = [&](int row, int c) {  // thread 0; the buffer region of the chunk must be free
    const T* src;
    int head, nvec, v0, v1;
    layout(row, src, head, nvec, v0, v1);
    const int p0 = c * kChunkVecs, p1 = min(v1 - v0, p0 + kChunkVecs);
    if (p1 <= p0) return;
    const uint32_t bytes = (uint32_t)(p1 - p0) * 16;
    mbar_expect_tx(&full[c], bytes);
    bulk_g2s(buf + p0, src + head + (long long)(v0 + p0) * V, bytes, &full[c]);
    pending |= 1u << c;
  };
  if (tid == 0 && team < M)
    for (int c = 0; c * kChunkVecs < per; ++c) load_chunk(team, c);
  bool alive = true;
  uint32_t phases = 0;  // bit c: parity of chunk c's next completion (a row may have one chunk fewer than another)
  for (int row = team, it = 0; row < M; row += teams, ++it) {
    const T* src;
    int head, nvec, v0, v1;
    layout(row, src, head, nvec, v0, v1);
    const int cnt = v1 - v0, tail = N - head - nvec * V;
    // elements outside the aligned middle: thread i < head + tail of rank 0 holds one
    const bool edge = rank == 0 && tid < head + tail;
    const int at = tid < head ? tid : nvec * V + tid;
    const float xe = edge ? (float)src[at] : 0.f;
    float m = -FLT_MAX, l = 0.f;
    if (edge) {  // m stays finite: a masked (-inf) element adds exp(-inf), and so do masked elements behind it
      m = fmaxf(xe, -FLT_MAX);
      l = exp_sub(xe, m);
    }
    for (int c = 0; c * kChunkVecs < cnt; ++c) {
      const int p0 = c * kChunkVecs, p1 = min(cnt, p0 + kChunkVecs);
      if (alive) alive = mbar_wait(&full[c], (phases >> c) & 1, status, DEV_TIMEOUT_TMA);
      if (alive) {
        phases ^= 1u << c;
        pending &= ~(1u << c);
      }
      for (int p = p0 + tid; p < p1; p += kRowThreads) {
        float f[V];
        unpack16<T>(buf[p], f);
        float cm = f[0];
#pragma unroll
        for (int k = 1; k < V; ++k) cm = fmaxf(cm, f[k]);
        if (cm > m) {
          l *= exp_sub(m, cm);
          m = cm;
        }
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < V; k += 2) s += exp_sub(f[k], m) + exp_sub(f[k + 1], m);
        l += s;
      }
    }
    auto over_warps = [&](float v, int which) {  // two sets of slots: no barrier behind the reads
      float* slot = red[it & 1][which];
      v = which == 0 ? warp_max(v) : warp_sum(v);
      if ((tid & 31) == 0) slot[tid >> 5] = v;
      __syncthreads();
      float r = slot[0];
#pragma unroll
      for (int k = 1; k < kRowThreads / 32; ++k) r = which == 0 ? fmaxf(r, slot[k]) : r + slot[k];  // fixed order
      return r;
    };
    float mx = over_warps(m, 0);
    float sum = over_warps(l * exp_sub(m, mx), 1);
    if (C > 1 && given_up) {  // the same for all threads: written ahead of the barriers of this row
      alive = false;
    } else if (C > 1) {
      // A peer sends its next row but one only after this CTA has sent its next, that is, read these slots.
      if (tid == 0) mbar_expect_tx(&met[it & 1], C * (uint32_t)sizeof(float2));
      if (tid < C) send_to_cta(&peers[it & 1][rank], mx, sum, &met[it & 1], (uint32_t)tid);
      if (!mbar_wait<true>(&met[it & 1], (it >> 1) & 1, status, DEV_TIMEOUT_TMA)) given_up = 1;
      float M2 = -FLT_MAX;
      for (int k = 0; k < C; ++k) M2 = fmaxf(M2, peers[it & 1][k].x);
      sum = 0.f;
      for (int k = 0; k < C; ++k) sum += peers[it & 1][k].y * exp_sub(peers[it & 1][k].x, M2);  // ascending rank
      mx = M2;
    }
    const float inv = 1.0f / sum;
    const int next = row + teams;
    T* dst = out + (long long)row * ld_out;
    if (edge) dst[at] = (T)(exp_sub(xe, mx) * inv);
    T* mid = dst + head + (long long)v0 * V;
    const bool vec = ((uintptr_t)mid & 15) == 0;
    for (int c = 0; c * kChunkVecs < per; ++c) {
      const int p0 = c * kChunkVecs, p1 = min(cnt, p0 + kChunkVecs);
      for (int p = p0 + tid; p < p1; p += kRowThreads) {
        float f[V];
        unpack16<T>(buf[p], f);
#pragma unroll
        for (int k = 0; k < V; ++k) f[k] = exp_sub(f[k], mx) * inv;
        if (vec) {
          uint4 q;
          if constexpr (sizeof(T) == 4) {
            q = make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
          } else {
            q = make_uint4(pack_f16x2(f[0], f[1]), pack_f16x2(f[2], f[3]), pack_f16x2(f[4], f[5]), pack_f16x2(f[6], f[7]));
          }
          __stcs(reinterpret_cast<uint4*>(mid) + p, q);
        } else {
#pragma unroll
          for (int k = 0; k < V; ++k) mid[(long long)p * V + k] = (T)f[k];
        }
      }
      __syncthreads();  // all reads of the chunk are done before the bulk copy overwrites it
      if (tid == 0 && next < M && alive) load_chunk(next, c);
    }
  }
  if (tid == 0)  // a wait ran out: copies under way must land before the CTA gives its shared memory back
    for (; pending; pending &= pending - 1)
      (void)mbar_wait(&full[__ffs(pending) - 1], (phases >> (__ffs(pending) - 1)) & 1, status, DEV_TIMEOUT_TMA);
  if (C > 1) {  // no peer sends any more, and what they have sent is there unless a wait ran out
    cluster_arrive_relaxed();
    cluster_wait();
    let_copies_land(&given_up);
  }
}

// ------------------------------------------------------------------ variant 1, any row
// VEC = elements per load (4 => Pack<T>, 1 => scalar).  CACHE = register-resident
// packs per thread; rows with more are re-read from global for the final pass.
template <typename T, int VEC, int CACHE>
__global__ void __launch_bounds__(kThreads) softmax_online_kernel(T* __restrict__ out, const T* __restrict__ in,
                                                                  int N, int M, long long ld_out, long long ld_in) {
  __shared__ float red[kWarps];
  grid_dependency_sync();
  const int tid = threadIdx.x;
  const int nvec = (N + VEC - 1) / VEC;  // VEC==4 only when N % 4 == 0
  const int nstep = (nvec + kThreads - 1) / kThreads;

  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    const T* src = in + (long long)row * ld_in;
    T* dst = out + (long long)row * ld_out;
    float cache[CACHE][VEC];
    float m = -FLT_MAX, l = 0.f;

    auto load = [&](int i, float* f) -> bool {
      const int p = tid + i * kThreads;
      if (p >= nvec) return false;
      if constexpr (VEC == 4) {
        Pack<T>::unpack(reinterpret_cast<const typename Pack<T>::type*>(src)[p], f);
      } else {
        f[0] = (float)src[p];
      }
      return true;
    };
    auto update = [&](const float* f) {
      float cm = f[0];
#pragma unroll
      for (int k = 1; k < VEC; ++k) cm = fmaxf(cm, f[k]);
      if (cm > m) {
        l *= exp_sub(m, cm);
        m = cm;
      }
#pragma unroll
      for (int k = 0; k < VEC; ++k) l += exp_sub(f[k], m);
    };

#pragma unroll
    for (int i = 0; i < CACHE; ++i)
      if (i < nstep && load(i, cache[i])) update(cache[i]);
    for (int i = CACHE; i < nstep; ++i) {
      float f[VEC];
      if (load(i, f)) update(f);
    }
    const float mg = block_max(m, red);
    const float inv = 1.0f / block_sum(l * exp_sub(m, mg), red);  // threads with no data: l = 0

    auto store = [&](int i, float* f) {
      const int p = tid + i * kThreads;
#pragma unroll
      for (int k = 0; k < VEC; ++k) f[k] = exp_sub(f[k], mg) * inv;
      if constexpr (VEC == 4) {
        reinterpret_cast<typename Pack<T>::type*>(dst)[p] = Pack<T>::pack(f);
      } else {
        dst[p] = (T)f[0];
      }
    };
#pragma unroll
    for (int i = 0; i < CACHE; ++i)
      if (i < nstep && tid + i * kThreads < nvec) store(i, cache[i]);
    for (int i = CACHE; i < nstep; ++i) {
      float f[VEC];
      if (load(i, f)) store(i, f);
    }
  }
}

// Teams (clusters of C CTAs) of softmax_long_kernel that run at once, with at most four CTAs per SM.  A team more would begin
// when another has done all its rows.  How many clusters fit depends on how many CTAs an SM takes: asked once per device for each.
template <typename T>
int long_teams(ctb_ctx* ctx, size_t smem, int C) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, softmax_long_kernel<T>, kRowThreads, smem);
  per_sm = std::max(1, std::min(4, per_sm));
  if (C == 1) return ctx->sm_count * per_sm;
  static int cached[16][kMaxCluster + 1][5] = {};
  int& n = cached[ctx->device & 15][C][per_sm];
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctx->sm_count * 4 / C * C);
    cfg.blockDim = dim3(kRowThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int m = 0;
    if (cudaOccupancyMaxActiveClusters(&m, softmax_long_kernel<T>, &cfg) != cudaSuccess || m < 1) {
      (void)cudaGetLastError();
      return std::max(1, ctx->sm_count * per_sm / C);
    }
    n = std::min(m, ctx->sm_count * per_sm / C);
  }
  return n;
}

template <typename T>
int launch(ctb_ctx* ctx, cudaStream_t st, T* out, const T* in, int N, int M, long long ldo, long long ldi,
           int variant, int tile_size) {
  const bool vec_ok = (N % 4 == 0) && (ldo % 4 == 0) && (ldi % 4 == 0) &&
                      ((uintptr_t)out % (4 * sizeof(T)) == 0) && ((uintptr_t)in % (4 * sizeof(T)) == 0);
  const size_t row_bytes = (size_t)N * sizeof(T);
  const bool bulk_ok = row_bytes % 16 == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)in % 16 == 0 &&
                       (ldo * sizeof(T)) % 16 == 0 && (ldi * sizeof(T)) % 16 == 0;
  constexpr int STAGES = 3, MAXV = 8;
  const bool fits = N <= 4 * kThreads * MAXV;
  if (variant == 0 && !bulk_ok)
    return fail(CTB_BAD_ALIGN,
                "ctb_softmax variant 0: rows must start on 16-byte boundaries and N*elemsize be a multiple of 16");
  if (variant == 0 && !fits)
    return fail(CTB_UNSUPPORTED, "ctb_softmax variant 0: N=%d exceeds the single-tile limit %d; use variant 1", N,
                4 * kThreads * MAXV);
  if (N <= 1024) {
    // both variants; a warp per CTA while that spreads the rows over more SMs
    const int warps = std::min(4, std::max(1, M / (2 * ctx->sm_count)));
    const int grid = std::min((M + warps - 1) / warps, ctx->sm_count * 16);
#define CTB_SOFTMAX_WARP(NE)                                                                                              \
  do {                                                                                                                    \
    if (vec_ok) launch_kernel(softmax_warp_kernel<T, NE, true>, grid, warps * 32, 0, st, 0, out, in, N, M, ldo, ldi);     \
    else launch_kernel(softmax_warp_kernel<T, NE, false>, grid, warps * 32, 0, st, 0, out, in, N, M, ldo, ldi);           \
  } while (0)
    if (N <= 128) CTB_SOFTMAX_WARP(4);
    else if (N <= 256) CTB_SOFTMAX_WARP(8);
    else if (N <= 512) CTB_SOFTMAX_WARP(16);
    else CTB_SOFTMAX_WARP(32);
#undef CTB_SOFTMAX_WARP
  } else if (bulk_ok && fits) {
    // Both variants: a row that fits the registers of one CTA is read once and written once whatever the chunk
    // size asks for; the chunk loop of the reference (examples/softmax.jl:48-100) only matters for longer rows.
    const int stage_bytes = (int)((row_bytes + 127) & ~size_t(127));
    const size_t smem = (size_t)STAGES * stage_bytes;
    auto k = softmax_staged_kernel<T, MAXV, STAGES>;
    cudaError_t e = allow_smem(k, (size_t)STAGES * 4 * kThreads * MAXV * sizeof(T));
    if (e != cudaSuccess) return cuda_fail(e, "ctb_softmax: shared memory opt-in");
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, smem);
    if (per_sm < 1) per_sm = 1;
    const int grid = min(M, ctx->sm_count * per_sm);
    launch_kernel(k, grid, kThreads, smem, st, 0, out, in, N, M, ldo, ldi, stage_bytes, ctx->dev_status);
  } else if (fits) {
    const int grid = std::min(M, ctx->sm_count * 8);
    if (N <= 8 * kThreads) launch_kernel(softmax_regs_kernel<T, 8>, grid, kThreads, 0, st, 0, out, in, N, M, ldo, ldi);
    else if (N <= 16 * kThreads) launch_kernel(softmax_regs_kernel<T, 16>, grid, kThreads, 0, st, 0, out, in, N, M, ldo, ldi);
    else launch_kernel(softmax_regs_kernel<T, 32>, grid, kThreads, 0, st, 0, out, in, N, M, ldo, ldi);
  } else if (row_bytes <= kMaxCluster * kLongBytes && (uintptr_t)in % sizeof(T) == 0) {
    int C = 1;
    while (row_bytes > C * kLongBytes) C *= 2;
    constexpr int V = 16 / (int)sizeof(T);
    const int per = (N / V + C - 1) / C;
    size_t smem = (size_t)per * 16;
    // Room for four CTAs on an SM is for many rows.  Where all rows run at once on up to three per SM, room for three is faster (f32
    // 150 x 8200 6.7 us with four, 6.0 with three, 150 x 27001 12.0 and 10.3; probably because the next kernel's CTAs come as early as
    // there is room and lie closer on some SMs than on others), unless a CTA has an SM to itself (f16 75 x 26000 7.2 and 8.1).
    if ((long long)M * C > ctx->sm_count && 10ll * M * C <= 27ll * ctx->sm_count) smem = std::max(smem, (size_t)60 * 1024);
    auto k = softmax_long_kernel<T>;
    cudaError_t e = allow_smem(k, kLongBytes);
    if (e != cudaSuccess) return cuda_fail(e, "ctb_softmax: shared memory opt-in");
    const int teams = std::min(M, long_teams<T>(ctx, smem, C));
    launch_kernel(k, teams * C, kRowThreads, smem, st, C, out, in, N, M, ldo, ldi, per, C, ctx->dev_status);
  } else {
    int per_sm = 8;
    const int grid = min(M, ctx->sm_count * per_sm);
    if (vec_ok)
      launch_kernel(softmax_online_kernel<T, 4, 8>, grid, kThreads, 0, st, 0, out, in, N, M, ldo, ldi);
    else
      launch_kernel(softmax_online_kernel<T, 1, 8>, grid, kThreads, 0, st, 0, out, in, N, M, ldo, ldi);
  }
  CTB_CHECK_LAUNCH("ctb_softmax launch");
  return CTB_OK;
}

}  // namespace

extern "C" int ctb_softmax(ctb_ctx* ctx, void* stream, void* output, const void* input, int64_t N, int64_t M,
                           int64_t ld_out, int64_t ld_in, int variant, int tile_size, int dtype) {
  CTB_CHECK_CTX(ctx);
  if (N <= 0 || M < 0 || N > INT32_MAX || M > INT32_MAX)
    return fail(CTB_BAD_ARG, "ctb_softmax: bad shape N=%lld M=%lld", (long long)N, (long long)M);
  if (ld_out < N || ld_in < N) return fail(CTB_BAD_ARG, "ctb_softmax: leading dimension smaller than N");
  if (variant != 0 && variant != 1) return fail(CTB_BAD_ARG, "ctb_softmax: variant must be 0 or 1");
  if (!is_pow2(tile_size)) return fail(CTB_UNSUPPORTED_TILE, "ctb_softmax: tile_size %d is not a power of two", tile_size);
  if (variant == 0 && tile_size < N)
    return fail(CTB_UNSUPPORTED_TILE, "ctb_softmax variant 0: tile_size %d must cover the row (N=%lld)", tile_size,
                (long long)N);
  if (M == 0) return CTB_OK;
  CTB_CHECK_DEV(output);
  CTB_CHECK_DEV(input);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == CTB_F32)
    return launch<float>(ctx, st, (float*)output, (const float*)input, (int)N, (int)M, ld_out, ld_in, variant, tile_size);
  if (dtype == CTB_F16)
    return launch<__half>(ctx, st, (__half*)output, (const __half*)input, (int)N, (int)M, ld_out, ld_in, variant, tile_size);
  return fail(CTB_BAD_ARG, "ctb_softmax: dtype must be CTB_F32 or CTB_F16");
}
