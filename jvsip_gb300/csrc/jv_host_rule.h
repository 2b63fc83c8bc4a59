// jv_host_rule.h -- which calls on host rows run faster on the host arrays
// themselves than through device copies (host arithmetic only, no CUDA headers).
#pragma once

#include <stddef.h>

namespace jv {

// Rows of `len` input elements `vs` apart, N the transform's length; `moved` the
// bytes that the kernel reads and writes over the host link, `staged` those of the
// copies (whole spans, gaps included).  kind 0: c2c, 1: R2C, 2: C2R.  Short rows make
// many small accesses to the link, and rows that overlap are read again; beyond a
// few MB the copies' bulk transfers win then.  Ratio of the direct time to the staged
// one at 2, 4, 8, 16 MB of single-precision rows: c2c of 64 points 0.54, 0.64, 1.07,
// 1.45, of 200 points 0.55, 0.69, 0.80, 0.89; R2C of 64 complex points 0.78, 1.06,
// 1.36, 1.59; C2R 0.65, 0.79, 0.99, 1.06; double precision c2c of 16 points 0.88, 1.16,
// 1.42, 1.69, of 24 points 0.55, 0.58, 0.77, 0.70; rows of 8 points 2 apart 1.02 at 1
// MB, 1.43 at 2 MB, of 1500 points 375 apart 0.51, 0.63, 0.86, 1.11, of 64 to 768
// points below 1 at any count.  Pitched views
// have no such line: the copies move their gaps too (5000 x 64 in rows of 256 points
// 39 us, 192 staged).
inline bool host_rows_pay(int kind, long N, long len, long vs, long nvec, bool f64, size_t moved, size_t staged) {
    const size_t MB = (size_t)1 << 20;
    if (staged > moved + moved / 4) return true;
    if (nvec > 1 && (vs < 0 ? -vs : vs) < len) return (N >= 24 && N < 1000) || moved <= (N < 24 ? MB : 8 * MB);
    if (f64) return N >= 24 || kind == 1 || moved <= 2 * MB;
    return N >= 200 || moved <= (kind == 1 ? 4 * MB : 8 * MB);
}

}  // namespace jv
