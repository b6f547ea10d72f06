// runs.cuh — x-runs of a class in row-aligned bit words (bit x & 31 of a row's
// word x / 32): run starts, the start of the run holding a bit, the piece of a run in a
// word.  Shared by the single-volume labelling and the batched atlas clustering.
#pragma once

namespace runs {
constexpr unsigned FULL = 0xffffffffu;

// x of the highest run start at or below bit b, or -1
__device__ __forceinline__ int last_start(unsigned starts, int x0, int b) {
    const unsigned hs = starts & (b == 31 ? FULL : (2u << b) - 1u);
    return hs ? x0 + 31 - __clz(hs) : -1;
}

// A row kernel's lane li of seg holds the class word c of its row that starts at x0: start (x) of the
// run holding the voxel before the word (-1: no run start before it).  carry_start / carry_word: the
// row's last run start and last class word of the chunks before this one (-1 / 0 before the first);
// all lanes call it
__device__ __forceinline__ int run_before(unsigned c, int x0, int li, int seg, int &carry_start, unsigned &carry_word) {
    const unsigned up = __shfl_up_sync(FULL, c, 1, seg), pc = li == 0 ? carry_word : up;
    const unsigned starts = c & ~((c << 1) | (pc >> 31));
    int incl = starts ? x0 + 31 - __clz(starts) : -1;
    for (int d = 1; d < seg; d <<= 1) {
        const int t = __shfl_up_sync(FULL, incl, d, seg);
        if (li >= d) incl = max(incl, t);
    }
    const int excl = __shfl_up_sync(FULL, incl, 1, seg);
    const int before = max(carry_start, li == 0 ? -1 : excl);
    carry_start = max(carry_start, __shfl_sync(FULL, incl, seg - 1, seg));
    carry_word = __shfl_sync(FULL, c, seg - 1, seg);
    return before;
}

// bits (x mask) of the piece of a run that starts at bit b of class word rem
__device__ __forceinline__ unsigned piece_at(unsigned rem, int b) {
    const unsigned ones = ~(rem >> b);
    const int len = ones ? __ffs(ones) - 1 : 32 - b;
    return (len == 32 ? FULL : (1u << len) - 1u) << b;
}

}  // namespace runs
