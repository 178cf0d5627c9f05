// solve_small.cu -- the solve kernels of systems with no more tile-rows than
// half-warps: CG on one-chunk matrices with its iterations in registers (up to
// 151,552 rows on 148 SMs), and every method as one cluster (up to 1,024 tile-rows).
// One block per SM is enough for them, so they take up to 128 registers.
#include "solver_dev.cuh"

namespace {

template <int LEN>
const void *resident_kernel(int mode, int lb)
{
    if (lb == 1)
        return mode == MODE_FP64 ? (const void *)k_solve<MODE_FP64, 1, MF_METHOD_CG, LEN, kVarResident>
                                 : (const void *)k_solve<MODE_MIXED, 1, MF_METHOD_CG, LEN, kVarResident>;
    return mode == MODE_FP64 ? (const void *)k_solve<MODE_FP64, 2, MF_METHOD_CG, LEN, kVarResident>
                             : (const void *)k_solve<MODE_MIXED, 2, MF_METHOD_CG, LEN, kVarResident>;
}

template <int LEN, int VAR>
const void *cluster_cg(int mode)
{
    return mode == MODE_FP64 ? (const void *)k_solve<MODE_FP64, 1, MF_METHOD_CG, LEN, VAR>
                             : (const void *)k_solve<MODE_MIXED, 1, MF_METHOD_CG, LEN, VAR>;
}

template <int LEN>
const void *cluster_kernel(int mode, int method, int rows_per_hw)
{
    if (method == MF_METHOD_BICGSTAB)
        return mode == MODE_FP64 ? (const void *)k_solve<MODE_FP64, 1, MF_METHOD_BICGSTAB, LEN, kVarCluster>
                                 : (const void *)k_solve<MODE_MIXED, 1, MF_METHOD_BICGSTAB, LEN, kVarCluster>;
    if constexpr (LEN > 0) {
        if (rows_per_hw == 2) return cluster_cg<LEN, kVarCluster2>(mode);
    }
    return cluster_cg<LEN, kVarCluster>(mode);
}

}  // namespace

const void *mf_solve_resident_kernel(int mode, int lb, int max_row)
{
    return max_row <= 5 ? resident_kernel<5>(mode, lb) : max_row <= 7 ? resident_kernel<7>(mode, lb)
                                                                     : resident_kernel<8>(mode, lb);
}

const void *mf_solve_cluster_kernel(int mode, int method, int max_row, int rows_per_hw)
{
    return max_row == 0 ? cluster_kernel<0>(mode, method, rows_per_hw)
           : max_row <= 5 ? cluster_kernel<5>(mode, method, rows_per_hw)
           : max_row <= 7 ? cluster_kernel<7>(mode, method, rows_per_hw)
                          : cluster_kernel<8>(mode, method, rows_per_hw);
}

int mf_small_chk_take() { return chk_take(); }
