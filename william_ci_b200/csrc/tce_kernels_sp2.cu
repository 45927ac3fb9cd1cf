// tce_kernels_sp2.cu -- the s/p tensor-core kernel (k_quartets_sp_tc,
// tce_kernels_tc.cuh) for the six classes with two p shells of one periodic
// direction (four power combinations per step loop), learned grid and system
// rule: 8 primitive quartets x 16 (shape 1) or 8 (shape 2) nodes per pass.
#include "tce_kernels_tc.cuh"

template <int NT, bool LG>
static int sp2_launch(const DevSys &S, int cls, const SArgs &A, int nsm, cudaStream_t st)
{
    switch (cls) {
    case 3: sp_tc_launch<1, 1, 0, 0, 1, NT, LG>(S, A, nsm, st); break;
    case 5: sp_tc_launch<1, 0, 1, 0, 1, NT, LG>(S, A, nsm, st); break;
    case 6: sp_tc_launch<0, 1, 1, 0, 1, NT, LG>(S, A, nsm, st); break;
    case 9: sp_tc_launch<1, 0, 0, 1, 1, NT, LG>(S, A, nsm, st); break;
    case 10: sp_tc_launch<0, 1, 0, 1, 1, NT, LG>(S, A, nsm, st); break;
    case 12: sp_tc_launch<0, 0, 1, 1, 1, NT, LG>(S, A, nsm, st); break;
    default: return TCE_ERR_UNSUPPORTED;
    }
    return TCE_OK;
}

int tce_sp2_launch(const DevSys &S, int cls, const SArgs &A, int shape, int nsm, cudaStream_t st)
{
    if (!A.item_rule) return shape == 1 ? sp2_launch<2, false>(S, cls, A, nsm, st) : sp2_launch<1, false>(S, cls, A, nsm, st);
    return shape == 1 ? sp2_launch<2, true>(S, cls, A, nsm, st) : sp2_launch<1, true>(S, cls, A, nsm, st);
}
