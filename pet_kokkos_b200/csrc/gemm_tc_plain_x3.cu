// The tensor-core GEMM with EPI_PLAIN in the formats of three parts.
#include "gemm_tc.cuh"

namespace petb {
template void run_format<EPI_PLAIN, FMT_F16X3>(Stream&, const GemmTask*, int);
template void run_format<EPI_PLAIN, FMT_F16X3_FULL>(Stream&, const GemmTask*, int);
}
