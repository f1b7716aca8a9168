// The tensor-core GEMM with EPI_SWIGLU.
#include "gemm_tc.cuh"

namespace petb {
template void run_tensor<EPI_SWIGLU>(Stream&, const GemmTask*, int);
}
