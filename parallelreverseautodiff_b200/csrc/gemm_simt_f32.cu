// The SIMT GEMM of gemm_simt.cuh for float.
#include "gemm_simt.cuh"

namespace prad {

template prad_status gemm_simt<float>(prad_ctx*, bool, bool, bool, int, int, int, double, const void*, int, const void*, int,
                                   double, void*, int, int, int64_t, int64_t, int64_t, const GemmEpilogue&);
template prad_status gemm_simt_backward<float>(prad_ctx*, bool, const void*, const void*, const void*, void*, void*, int, int, int, bool,
                                            double, const GemmEpilogue&);

}  // namespace prad
