// Blocks of an expert's slots and where their accumulators lie (moe_ffn.cu).  Plain integers, so that a host compiler takes it too.
#pragma once
#ifdef __CUDACC__
#define CTB_PLACE __host__ __device__ __forceinline__
#else
#define CTB_PLACE inline
#endif

namespace ctb_internal {

constexpr int kMmaSlots = 256;       // MMA N
constexpr int kMaxBlockSlots = 320;  // slots of a block: two MMAs above kMmaSlots
// Blocks that an expert's slots are cut into.  A k-block costs a pair about 330 ns up to 224 slots, whatever their number, and
// the MMA's 1.45 ns per slot above: blocks of 226 slots and more are cheap, and one of up to 320 is cheaper than two of half of it.
// (ring: the accumulators of moe_pair_gemm_kernel may take more than half of the columns.)
constexpr CTB_PLACE int blocks_for(bool ring, int slots) {
  const int n = (slots + kMmaSlots - 1) / kMmaSlots;
  return ring && n > 1 && slots < n * 226 && slots <= (n - 1) * kMaxBlockSlots ? n - 1 : n;
}

// Where a block's accumulators lie in the 512 TMEM columns, which are a ring: slot s of the block in column
// (col + s) mod 512, col a multiple of 32.  The slots are taken by at most two MMAs: [0, first) and [first, n).
struct Place {
  int col, first, next, skipped;  // next: where the next block may start
};
constexpr int kParts = 6;  // leading blocks of 32 columns of an item that the next one may need
template <bool RING>
CTB_PLACE Place place(int at, int n) {
  if (!RING) return {at, n, at ^ 256, 0};  // no block above 256 slots: two halves in turn
  const int n32 = (n + 31) & ~31, room = 512 - at;
  Place r;
  // an MMA takes at most kMmaSlots: columns before or behind the end of the ring stay unused where a part would be larger
  r.skipped = n32 <= room ? 0 : room > kMmaSlots ? room - kMmaSlots : n - room > kMmaSlots ? room : 0;
  r.col = (at + r.skipped) & 511;
  const int left = 512 - r.col;
  r.first = n32 > left ? left : n > kMmaSlots ? ((n / 2 + 15) & ~15) : n;
  r.next = (r.col + n32) & 511;
  return r;
}

}  // namespace ctb_internal
