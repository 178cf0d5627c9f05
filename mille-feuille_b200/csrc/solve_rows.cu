// solve_rows.cu -- the solve kernels of one-chunk matrices: every tile-row is one
// slice of 16 rows x 8 entries (5- and 7-point stencils and the like).  By the
// longest row: 5, 7 or 8 entries are loaded, gathered and multiplied.
#include "solver_dev.cuh"

namespace {

template <int LEN>
const void *rows_kernel(int mode, int method)
{
    if (method == MF_METHOD_BICGSTAB)
        return mode == MODE_FP64 ? (const void *)k_solve<MODE_FP64, 2, MF_METHOD_BICGSTAB, LEN, kVarGrid>
                                 : (const void *)k_solve<MODE_MIXED, 2, MF_METHOD_BICGSTAB, LEN, kVarGrid>;
    return mode == MODE_FP64 ? (const void *)k_solve<MODE_FP64, 2, MF_METHOD_CG, LEN, kVarGrid>
                             : (const void *)k_solve<MODE_MIXED, 2, MF_METHOD_CG, LEN, kVarGrid>;
}

}  // namespace

const void *mf_solve_rows_kernel(int mode, int method, int max_row)
{
    return max_row <= 5 ? rows_kernel<5>(mode, method) : max_row <= 7 ? rows_kernel<7>(mode, method)
                                                                     : rows_kernel<8>(mode, method);
}

int mf_rows_chk_take() { return chk_take(); }
