// jv_tma_box.h -- boxes of the TMA-staged column tiles (host arithmetic only, no
// CUDA headers).
#pragma once

namespace jv {

// A tile of vpb transforms of N points, 2*vpb scalars of `esz` bytes to a row, as
// `boxes` boxes of `rows` rows each, one behind the other in the tile's shared
// memory (ld rows).  A box is at most 256 rows and its bytes a multiple of 128, the
// alignment of a tensor copy's shared-memory address, for every vpb: 6 transforms of
// 4-byte scalars take rows by eights.  False when the boxes do not fit.
inline bool tma_boxes(long N, long vpb, long esz, long ld, long *boxes, long *rows) {
    long q = 128;  // rows whose bytes are a multiple of 128: 128 / gcd(128, bytes of a row)
    while (q > 1 && (q / 2 * vpb * 2 * esz) % 128 == 0) q /= 2;
    const long nb = (N + 255) / 256;
    *rows = ((N + nb - 1) / nb + q - 1) / q * q;
    *boxes = nb;
    return *rows <= 256 && nb * *rows <= ld;
}

}  // namespace jv
