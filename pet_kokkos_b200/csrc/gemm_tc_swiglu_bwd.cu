// The tensor-core GEMM with EPI_SWIGLU_BWD.
#include "gemm_tc.cuh"

namespace petb {
template void run_tensor<EPI_SWIGLU_BWD>(Stream&, const GemmTask*, int);
}
