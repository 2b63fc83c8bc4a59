// jv_dif_fixt2.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// the k-omega pipeline's tapered R2C rows, longer ones.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_taper_2(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_taper<__VA_ARGS__>());
    JV_DIF_R2C_2(X)
#undef X
}
}  // namespace jv
