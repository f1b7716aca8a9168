// The tensor-core GEMM with EPI_PLAIN.
#include "gemm_tc.cuh"

namespace petb {
template void run_tensor<EPI_PLAIN>(Stream&, const GemmTask*, int);
}
