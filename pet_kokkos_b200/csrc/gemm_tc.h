// What the parts of the tensor-core GEMM share (gemm_tc.cuh has the kernel, gemm_tc_<epilogue>.cu its instances).
#pragma once

#include <cuda.h>

#include "gemm.h"

namespace petb {

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// What the tensor-core path needs of one device: its SM count and the driver's tensor-map encoder (the same function for every device). One per device ordinal,
// built on first use with that device current.
struct TensorState {
  EncodeFn encode = nullptr;
  int sms = 0;
  bool ok = false;
};
TensorState& tensor_state();

// A GEMM and the packed weight it reads.
struct GemmTask {
  GemmArgs a;
  PackedB w;
};

// One or two GEMMs of one epilogue and operand format; two go as one launch where that is expected to end first.
template <int EPI>
void run_tensor(Stream& st, const GemmTask* q, int n);
extern template void run_tensor<EPI_PLAIN>(Stream&, const GemmTask*, int);
extern template void run_tensor<EPI_SILU>(Stream&, const GemmTask*, int);
extern template void run_tensor<EPI_SWIGLU>(Stream&, const GemmTask*, int);
extern template void run_tensor<EPI_SILU_BWD>(Stream&, const GemmTask*, int);
extern template void run_tensor<EPI_SWIGLU_BWD>(Stream&, const GemmTask*, int);
extern template void run_tensor<EPI_COMPRESS>(Stream&, const GemmTask*, int);

}  // namespace petb
