"""Where the MoE kernels put the accumulators of an expert's blocks (csrc/moe_place.h), compiled for the host: every start in the ring of 512
columns and every two blocks in a row."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECK = r"""
#include <cstdio>
#include <cstring>
#include "moe_place.h"
using namespace ctb_internal;
#define REQUIRE(c) do { if (!(c)) { std::printf("%s: at %d, blocks of %d and %d\n", #c, at, n, n2); return 1; } } while (0)
// marks the columns of a block with `who`; counts those that were `before`, and leaves the last column of them in *last
static int fill(unsigned char* col, const Place& p, int n, int who, int before, int origin, int* last) {
  int taken = 0;
  for (int s = 0; s < n; ++s) {
    unsigned char& c = col[(p.col + s) & 511];
    if (c == before) { ++taken; const int at = ((p.col + s) - origin) & 511; if (at > *last) *last = at; }
    c = (unsigned char)who;
  }
  return taken;
}
int main() {
  for (int at = 0; at < 512; at += 32)
    for (int n = 16; n <= kMaxBlockSlots; n += 16)
      for (int n2 = 16; n2 <= kMaxBlockSlots; n2 += 16) {
        unsigned char col[512];
        std::memset(col, 0, sizeof col);
        const Place a = place<true>(at, n), b = place<true>(a.next, n2);
        const int sizes[2] = {n, n2};
        const Place* places[2] = {&a, &b};
        for (int k = 0; k < 2; ++k) {  // two MMAs at most, neither across the end of the ring nor above 256 slots, in steps of 16
          const Place& p = *places[k];
          const int rest = sizes[k] - p.first;
          REQUIRE(p.col % 32 == 0 && p.next % 32 == 0 && p.first % 16 == 0 && rest % 16 == 0 && p.first > 0 && rest >= 0);
          REQUIRE(p.first <= kMmaSlots && rest <= kMmaSlots && p.col + p.first <= 512);
          REQUIRE(rest == 0 || ((p.col + p.first) & 511) + rest <= 512);
          REQUIRE(p.next == ((p.col + ((sizes[k] + 31) & ~31)) & 511));
        }
        REQUIRE(b.col == ((a.next + b.skipped) & 511));
        int none = -1, last = -1;
        fill(col, a, n, 1, 9, 0, &none);
        const int taken = fill(col, b, n2, 2, 1, a.col, &last);
        // the second block waits for the first `shared` blocks of 32 columns of the first one, of which kParts have a barrier
        const int shared = (((n + 31) & ~31) + b.skipped + ((n2 + 31) & ~31) - 512) / 32;
        REQUIRE(shared <= kParts);
        REQUIRE(taken == 0 || last < shared * 32);
      }
  for (int slots = 0; slots <= 70000; ++slots) {  // equal blocks of whole 16 slots fit
    const int at = slots, n = blocks_for(true, slots), n2 = blocks_for(false, slots);
    REQUIRE((slots == 0) == (n == 0) && n <= n2 && n2 == (slots + kMmaSlots - 1) / kMmaSlots);
    if (n) REQUIRE((((slots + n - 1) / n + 15) & ~15) <= kMaxBlockSlots && (((slots + n2 - 1) / n2 + 15) & ~15) <= kMmaSlots);
  }
  return 0;
}
"""


def test_accumulators_in_the_ring(tmp_path):
    (tmp_path / "check.cpp").write_text(CHECK)
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "cutile.jl_b200", "csrc"), str(tmp_path / "check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
