// The tensor-core GEMM with EPI_COMPRESS.
#include "gemm_tc.cuh"

namespace petb {
template void run_tensor<EPI_COMPRESS>(Stream&, const GemmTask*, int);
}
