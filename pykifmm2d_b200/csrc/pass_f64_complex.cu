// pass_f64_complex.cu -- P2M and the L2P + P2P at the sources for complex
// densities (iscomplex=True, class_fmm.py:174): the kernels of pass_f64.cuh on
// double2 charges and sums.  In a file of its own to build beside pass_f64.cu.
#include "pass_f64.cuh"

namespace kifmm {

void launch_leaf_eval_dc(kifmm_plan *P, const PassArgs &A, int check_self) {
    if (P->kern.kind == KIFMM_KERNEL_LAPLACE)
        launch_leaf_eval<KIFMM_KERNEL_LAPLACE, true, false>(P, A, check_self);
    else if (P->kern.kind == KIFMM_KERNEL_MOD_HELMHOLTZ)
        launch_leaf_eval<KIFMM_KERNEL_MOD_HELMHOLTZ, true, false>(P, A, check_self);
    else launch_leaf_eval<KIFMM_KERNEL_HELMHOLTZ, true, false>(P, A, check_self);
}
void launch_p2m_dc(kifmm_plan *P, const PassArgs &A) {
    KIFMM_REQUIRE(P->Qc <= 32, KIFMM_ERR_ARG, "complex form: Nequiv above 32");
    if (P->kern.kind == KIFMM_KERNEL_LAPLACE) launch_p2m_kind<KIFMM_KERNEL_LAPLACE, true>(P, A);
    else if (P->kern.kind == KIFMM_KERNEL_MOD_HELMHOLTZ) launch_p2m_kind<KIFMM_KERNEL_MOD_HELMHOLTZ, true>(P, A);
    else launch_p2m_kind<KIFMM_KERNEL_HELMHOLTZ, true>(P, A);
}

}  // namespace kifmm
