// The tensor-core GEMM with EPI_SILU_BWD.
#include "gemm_tc.cuh"

namespace petb {
template void run_tensor<EPI_SILU_BWD>(Stream&, const GemmTask*, int);
}
