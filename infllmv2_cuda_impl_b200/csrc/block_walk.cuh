// Walks over the key blocks that a tile of 8 query tokens visits: the set bits of the union of its
// tokens' block-mask rows, highest block first.
#pragma once
#include "common.cuh"

namespace ifv2 {

// One thread's walk (the copy warp's).
struct BlockWalk {
  const unsigned long long* words;
  int w;
  unsigned long long cur;
  __device__ BlockWalk(const unsigned long long* u, int nwords) : words(u), w(nwords), cur(0) {}
  __device__ int next() {
    while (cur == 0ull) {
      if (w == 0) return -1;
      cur = words[--w];
    }
    const int b = 63 - __clzll(cur);
    cur &= ~(1ull << b);
    return w * 64 + b;
  }
};

// The softmax warps' walk: 32 blocks at a time, one per lane, with the tokens that selected them.  A
// warp owns the 32 rows of two tokens, so a token's selection of 32 blocks is one ballot.  (Walking
// block by block in every thread, with its own mask word, cost ~350 of the ~1570 clocks that a softmax
// warp of the forward kernel spends on a block: long chains of 64-bit bit arithmetic in front of the
// wait for the scores.)  Every lane must make the calls.
struct WalkBatch {
  int blk;                 // lane l: number 32 n + l of the walk
  uint32_t sel;            // bit l: this lane's token selected it
  uint32_t any;            // bit l: one of the warp's tokens did
  // umask: union mask in shared memory; masked: token selections come from row0 / row1 (this warp's two
  // tokens, null = not a token of the sequence), otherwise every block counts as selected
  __device__ void refill(const unsigned long long* umask, int words, int i0, bool masked,
                         const unsigned long long* row0, const unsigned long long* row1, int lane) {
    const int target = i0 + lane;
    int before = 0;
    blk = -1;
    for (int top = words - 1; top >= 0 && before <= i0 + 31; top -= 32) {
      const unsigned long long mine = top - lane >= 0 ? umask[top - lane] : 0ull;
      const int cnt = __popcll(mine);
      int incl = cnt;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += up;
      }
      const int excl = incl - cnt, total = __shfl_sync(0xFFFFFFFFu, incl, 31);
      const bool here = target >= before && target < before + total;
      const int r = here ? target - before : 0;
      int src = 0;                               // last word that starts at or below block r of the chunk
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1)
        if (__shfl_sync(0xFFFFFFFFu, excl, src + d) <= r) src += d;
      unsigned long long x = __shfl_sync(0xFFFFFFFFu, mine, src);
      // r counts from the word's highest set bit: turn it into the number of set bits below
      int rank = __popcll(x) - 1 - (r - __shfl_sync(0xFFFFFFFFu, excl, src)), pos = 0;
#pragma unroll
      for (int d = 32; d >= 1; d >>= 1) {
        const int low = __popcll(x & ((1ull << d) - 1ull));
        if (rank >= low) { rank -= low; pos += d; x >>= d; }
      }
      if (here) blk = (top - src) * 64 + pos;
      before += total;
    }
    bool s0 = false, s1 = false;
    if (blk >= 0) {
      s0 = !masked || (row0 != nullptr && ((__ldg(row0 + (blk >> 6)) >> (blk & 63)) & 1ull));
      s1 = !masked || (row1 != nullptr && ((__ldg(row1 + (blk >> 6)) >> (blk & 63)) & 1ull));
    }
    const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, s0), b1 = __ballot_sync(0xFFFFFFFFu, s1);
    sel = lane < 16 ? b0 : b1;
    any = b0 | b1;
  }
};

}  // namespace ifv2
