// The tensor-core GEMM with EPI_PLAIN, but for the formats of three parts.
#include "gemm_tc.cuh"

namespace petb {
template void run_tensor<EPI_PLAIN>(Stream&, const GemmTask*, int);
}
