// jv_dif_fixq1.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// c2c rows of lengths with one factor 7, 11 or 13, up to 1500 points.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_rows_1(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_real<DIF_C2C, __VA_ARGS__>());
    JV_DIF_ROWS_1(X)
#undef X
}
}  // namespace jv
