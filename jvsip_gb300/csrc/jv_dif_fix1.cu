// jv_dif_fix1.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// c2c rows and column tiles up to 600 points.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_c2c_1(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_c2c<__VA_ARGS__>());
    JV_DIF_LENGTHS_1(X)
#undef X
}
}  // namespace jv
