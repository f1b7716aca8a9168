// The tensor-core GEMM with EPI_SILU.
#include "gemm_tc.cuh"

namespace petb {
template void run_tensor<EPI_SILU>(Stream&, const GemmTask*, int);
}
