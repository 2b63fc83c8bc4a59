// jv_kern_f64.cu -- double-precision instances of the general kernels (c2c
// shared-memory kernel, global-memory path, capacity query, helper kernels of
// the real long transforms); the real
// transforms' shared-memory kernels are in jv_kern_f64r.cu.
#include "jv_launch.cuh"

namespace jv {
bool launch_smem_fold_f64(const Job &j, cudaStream_t s);
static bool radices_2k(const Job &j) {
    for (int i = 0; i < j.npass; i++)
        if (j.radix[i] & (j.radix[i] - 1)) return false;
    return j.npass > 0;
}
bool launch_smem_f64(const Job &j, cudaStream_t s) {
    if (j.kind == K_C2C && j.cin.cst == 1 && j.cout.cst == 1) return launch_smem_split_f64(j, s);
    if (j.kind == K_C2C && radices_2k(j)) return launch_smem_fold_f64(j, s);
    if (j.kind == K_C2C) return launch_smem_t<double, K_C2C>(j, s);
    return launch_smem_real_f64(j, s);
}
bool launch_global_f64(const Job &j, cudaStream_t s) { return launch_global_t<double>(j, s); }
long smem_max_len_f64(int kind) { return smem_len_limit<double>(kind); }
bool launch_r2c_pairs_f64(void *z, long es, long vs, long N, long nvec, int has_scale, double scale,
                         const void *thalf, cudaStream_t s) {
    return launch_r2c_pairs_t<double>(z, es, vs, N, nvec, has_scale, scale, thalf, s);
}
bool launch_c2r_unsplit_f64(const Job &j, void *ydst, cudaStream_t s) { return launch_c2r_unsplit_t<double>(j, ydst, s); }
bool launch_c2r_unpack_f64(const Job &j, const void *y, cudaStream_t s) { return launch_c2r_unpack_t<double>(j, y, s); }
}  // namespace jv
