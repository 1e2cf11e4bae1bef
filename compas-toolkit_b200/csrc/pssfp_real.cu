// pssfp_real.cu — instantiations of the real-RF pSSFP value kernels (pssfp_real.cuh), one per layout of
// pssfp.cu.
#include "compas/compas.h"
#include "pssfp_real.cuh"

namespace compas {

const PssfpRealKernels& pssfp_real_kernels(int ZT, int GZ) {
#define COMPAS_REAL(ZT, GZ)                                                                        \
    {ZT, GZ, kernels::pssfp_real_kernel<ZT, GZ, false>, kernels::pssfp_real_queue_kernel<ZT, GZ, false>}
    static const PssfpRealKernels table[] = {
        COMPAS_REAL(1, 1), COMPAS_REAL(2, 1), COMPAS_REAL(4, 1), COMPAS_REAL(8, 1), COMPAS_REAL(9, 1), COMPAS_REAL(10, 1),
        COMPAS_REAL(6, 2), COMPAS_REAL(18, 2), COMPAS_REAL(2, 4), COMPAS_REAL(4, 4), COMPAS_REAL(6, 4), COMPAS_REAL(8, 4),
        COMPAS_REAL(9, 4), COMPAS_REAL(10, 4), COMPAS_REAL(12, 4), COMPAS_REAL(4, 8), COMPAS_REAL(5, 8), COMPAS_REAL(8, 8),
        COMPAS_REAL(3, 16), COMPAS_REAL(1, 32), COMPAS_REAL(2, 32),
    };
#undef COMPAS_REAL
    for (const auto& k : table)
        if (k.ZT == ZT && k.GZ == GZ) return k;
    COMPAS_ERROR("no real-RF kernels for this pSSFP layout");
}

}  // namespace compas
