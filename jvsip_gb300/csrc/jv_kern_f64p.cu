// jv_kern_f64p.cu -- double-precision c2c instance of the shared-memory kernel
// for schedules of radices 2^k, whose twiddles and constants are folded into the
// additions (tw_bfly).  An instance of its own: with the folded codelets beside
// the others one kernel spilled less and was still slower at most lengths with
// factors 3, 5 and 7 (us: 21 points 6.1 -> 6.8, 100 12.9 -> 13.6, 216 15.2 -> 16.1,
// 2400 67.3 -> 71.9), which keep the kernel with products.
#include "jv_launch.cuh"

namespace jv {
bool launch_smem_fold_f64(const Job &j, cudaStream_t s) { return launch_smem_t<double, KX_C2C_FOLD>(j, s); }
}  // namespace jv
