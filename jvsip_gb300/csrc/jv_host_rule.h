// jv_host_rule.h -- which calls on host rows run faster on the host arrays
// themselves than through device copies (host arithmetic only, no CUDA headers).
#pragma once

#include <stddef.h>

namespace jv {

// Rows of `len` input elements `vs` apart, N the transform's length, `moved` the
// bytes that the kernel reads and writes over the host link.  Short rows make many
// small accesses to it, and rows that overlap are read again; beyond a few MB the
// copies' bulk transfers win then.  Ratio of the direct time to the staged one at 2,
// 4, 8, 16 MB of single-precision c2c rows: 64 points 0.54, 0.64, 1.07, 1.45, 200
// points 0.55, 0.69, 0.80, 0.89; R2C of 64 complex points 0.78, 1.06, 1.36, 1.59;
// double precision 16 points 0.88, 1.16, 1.42, 1.69, 24 points 0.55, 0.58, 0.77,
// 0.70; overlapping rows of 8 points 1.43 at 2 MB, 1.02 at 1 MB, of 4096 points 0.68,
// 0.92, 1.10.
inline bool host_rows_pay(long N, long len, long vs, long nvec, bool f64, size_t moved) {
    const bool overlap = nvec > 1 && (vs < 0 ? -vs : vs) < len;
    const bool brief = N < (f64 ? 24 : 200);
    if (overlap) return moved <= (brief ? (size_t)1 << 20 : (size_t)4 << 20);
    return !brief || moved <= (size_t)2 << 20;
}

}  // namespace jv
