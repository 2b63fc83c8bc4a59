// jv_dif_tile.h -- transforms and threads of the in-place mixed-radix kernel's
// column tiles (host arithmetic only, no CUDA headers).
//
// Thread i of a tile of V = 2^lgv transforms takes transform i mod V, and the
// loops over butterflies start at i / V and advance by threads / V: the threads
// are a multiple of V and at least V, whatever tile was asked for.  With fewer
// the loops would not advance; with a remainder two threads would take one
// butterfly, which the in-place passes must not do.
#pragma once

namespace jv {

constexpr int kDifColLgMax = 9;  // 512 transforms: the most threads of a tile of 16384 points and fewer

// log2 of the transforms per tile where `tuned` are asked for, of nvec in all
inline int dif_col_tuned(long tuned, long nvec) {
    int lgv = 0;
    while (lgv < kDifColLgMax && (2L << lgv) <= tuned && (1L << lgv) < nvec) lgv++;
    return lgv;
}

// log2 of the transforms per tile, from lgv down, while twice as many tiles still
// have an SM each
inline int dif_col_narrow(int lgv, long nvec, long sms) {
    while (lgv > 0 && 2 * (((nvec - 1) >> lgv) + 1) <= sms) lgv--;
    return lgv;
}

// threads of a tile of 2^lgv transforms of N points: about 16 points each (8 where
// every tile has an SM to itself: `few`), 64 to 512, and 1024 for single-precision
// tiles that ask for that many
inline long dif_col_threads(long N, int lgv, bool f32, bool few) {
    const long V = 1L << lgv, unit = V < 32 ? 32 : V, pts = few ? 8 : 16;
    const long most = f32 && (few || V * N > 16384) ? 1024 : 512;
    const long want = V * N / pts < 64 ? 64 : V * N / pts;
    const long n = (want + unit - 1) / unit * unit;
    return n < most ? n : most;
}

// rounded up to the batching form's block sizes (multiples of 64, still of V)
inline int dif_batch_threads(int nthr) { return (nthr + 63) / 64 * 64; }

}  // namespace jv
