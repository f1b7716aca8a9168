// The tensor-core GEMM's packing, row maxima and entry points: see gemm_tc.cuh.
#include "gemm_tc.cuh"

namespace petb {

namespace {

// ---- packing, row maxima ----------------------------------------------------------------------

// What undoes the scale of each row of a weight, a block per row (past the last one: zeros); and whether more than a quarter of a
// row's values (and more than eight; zeros do not count) lie below 2^-7 of its largest. Of 256 normal values some 2 % do.
__global__ void k_row_unscale(const float* __restrict__ W, size_t ld_r, size_t ld_k, int rows, int K, uint16_t* __restrict__ unscale,
                              int* __restrict__ spread) {
  __shared__ uint32_t s_max;
  __shared__ int s_low;
  const int r = blockIdx.x;
  if (threadIdx.x == 0) s_max = 0, s_low = 0;
  __syncthreads();
  float m = 0.f;
  if (r < rows)
    for (int k = threadIdx.x; k < K; k += blockDim.x) m = fmaxf(m, fabsf(W[r * ld_r + k * ld_k]));
  const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if ((threadIdx.x & 31) == 0) atomicMax(&s_max, most);
  __syncthreads();
  if (threadIdx.x == 0) unscale[r] = r < rows ? __float_as_uint(unscale_of(s_max)) >> 16 : 0;
  if (r >= rows) return;
  const float low = __uint_as_float(s_max) * 0.0078125f;
  int n = 0;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const float x = fabsf(W[r * ld_r + k * ld_k]);
    n += x < low && x > 0.f;
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) atomicAdd(&s_low, n);
  __syncthreads();
  if (threadIdx.x == 0 && s_low > 8 && 4 * s_low > K) *spread = 1;
}

// Whether a column's values all lie 2^-4 and more below their rows' scales. 32 columns a block, 32 rows at a time. (A column of
// sixteen normal values does with a probability of 1e-9.)
__global__ void k_column_spread(const float* __restrict__ W, size_t ld_r, size_t ld_k, int rows, int K, const uint16_t* __restrict__ unscale,
                                int* __restrict__ spread) {
  __shared__ float s_max[32][33];
  const int k = blockIdx.x * 32 + threadIdx.x;
  float m = 0.f;
  if (k < K)
    for (int r = threadIdx.y; r < rows; r += 32) m = fmaxf(m, fabsf(W[r * ld_r + k * ld_k]) / __uint_as_float(uint32_t(unscale[r]) << 16));
  s_max[threadIdx.y][threadIdx.x] = m;
  __syncthreads();
  if (threadIdx.y != 0 || k >= K) return;
  for (int r = 1; r < 32; ++r) m = fmaxf(m, s_max[r][threadIdx.x]);
  if (m > 0.f && m < 2048.f) *spread = 1;
}

template <int FMT>
__global__ void k_pack_weight(const float* __restrict__ W, size_t ld_r, size_t ld_k, int rows, int K, int Kp, const uint16_t* __restrict__ unscale,
                              uint16_t* __restrict__ main, uint16_t* __restrict__ low) {
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= size_t(rows) * (Kp / 2)) return;
  const int r = int(i / (Kp / 2)), k = 2 * int(i % (Kp / 2));
  const float x = k < K ? W[r * ld_r + k * ld_k] : 0.f, y = k + 1 < K ? W[r * ld_r + (k + 1) * ld_k] : 0.f;
  uint32_t h, m, l;
  split2<FMT>(x, y, scales_rows(FMT) ? 1.f / __uint_as_float(uint32_t(unscale[r]) << 16) : 1.f, h, m, l);  // (powers of two: exact)
  if (FMT == FMT_TF32X2 || FMT == FMT_TF32) {
    *reinterpret_cast<float2*>(reinterpret_cast<float*>(main) + size_t(r) * Kp + k) = make_float2(x, y);
    if (FMT == FMT_TF32X2) *reinterpret_cast<float2*>(reinterpret_cast<float*>(low) + size_t(r) * Kp + k) = make_float2(tf32_low(x), tf32_low(y));
    return;
  }
  if (FMT == FMT_BF16 || FMT == FMT_F16) {
    *reinterpret_cast<uint32_t*>(main + size_t(r) * Kp + k) = h;
    return;
  }
  const size_t at = size_t(r) * Kp * 2 + (k / 32) * 64 + k % 32;
  *reinterpret_cast<uint32_t*>(main + at) = h, *reinterpret_cast<uint32_t*>(main + at + 32) = m;
  if (FMT == FMT_F16X3) *reinterpret_cast<uint32_t*>(low + size_t(r) * Kp + k) = l;
}

__global__ void __launch_bounds__(256) k_row_max(uint32_t* __restrict__ mx, const float* __restrict__ x, int ld, int R, int D4) {
  after_previous();
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= R) return;
  float m = 0.f;
  for (int c = lane; c < D4; c += 32) {
    const float4 v = ld4(x + size_t(r) * ld + 4 * c);
    m = fmaxf(m, max_abs4(v.x, v.y, v.z, v.w));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) mx[r] = __float_as_uint(m);
}

}  // namespace

TensorState& tensor_state() {
  static PerDevice<TensorState> table;
  int dev = 0;
  cudaGetDevice(&dev);
  return table.get(dev, [dev](TensorState& s) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn) return;
    int major = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, dev);
    if (major != 10 || s.sms <= 0) return;
    s.encode = reinterpret_cast<EncodeFn>(fn);
    s.ok = true;
  });
}


PackedB pack_weight(cudaStream_t s, Format fmt, const float* W, size_t ld_r, size_t ld_k, int rows, int K, uint16_t* out, uint16_t* unscale) {
  PackedB w;
  w.fmt = fmt, w.Kp = packed_k(K), w.main = out, w.unscale = unscale;
  uint16_t* low = three_parts(fmt) || fmt == FMT_TF32X2 ? out + 2 * size_t(rows) * w.Kp : nullptr;
  w.low = low;
  if (rows <= 0 || K <= 0) return w;
  const unsigned blocks = unsigned(cdiv((long long) rows * (w.Kp / 2), 256));
  if (scales_rows(fmt)) {
    int* spread = reinterpret_cast<int*>(unscale + unscale_halves(rows) - 8);
    PETB_CUDA(cudaMemsetAsync(spread, 0, 16, s));
    k_row_unscale<<<unsigned(unscale_halves(rows) - 8), 128, 0, s>>>(W, ld_r, ld_k, rows, K, unscale, spread);
    if (fmt == FMT_F16X3 && rows >= 16) k_column_spread<<<cdiv(K, 32), dim3(32, 32), 0, s>>>(W, ld_r, ld_k, rows, K, unscale, spread);
  }
  auto kernel = three_parts(fmt) ? k_pack_weight<FMT_F16X3> : fmt == FMT_F16X2 ? k_pack_weight<FMT_F16X2> : fmt == FMT_F16 ? k_pack_weight<FMT_F16>
                : fmt == FMT_BF16 ? k_pack_weight<FMT_BF16> : fmt == FMT_TF32X2 ? k_pack_weight<FMT_TF32X2> : k_pack_weight<FMT_TF32>;
  kernel<<<blocks, 256, 0, s>>>(W, ld_r, ld_k, rows, K, w.Kp, unscale, out, low);
  PETB_CUDA(cudaGetLastError());
  return w;
}

bool values_spread(const PackedB& w, int rows) {
  if (w.fmt != FMT_F16X3 || rows <= 0) return false;
  int spread = 0;
  PETB_CUDA(cudaMemcpy(&spread, w.unscale + unscale_halves(rows) - 8, sizeof(int), cudaMemcpyDeviceToHost));
  return spread != 0;
}

void full_if_spread(PackedB& w, int rows) {
  if (values_spread(w, rows)) w.fmt = FMT_F16X3_FULL;
}

void row_max(Stream& st, uint32_t* mx, const float* x, int ld, int R, int D) {
  if (R <= 0) return;
  launch(st, k_row_max, cdiv((long long) R * 32, 256), 256, 0, mx, x, ld, R, D / 4);
  PETB_LAUNCH_CHECK(st);
}

bool tensor_gemm_available() { return tensor_state().ok; }

// Whether a tensor-core kernel takes this GEMM: a packed weight, and rows that TMA can address (16-byte aligned).
bool gemm_tensor_usable(const Stream& st, const GemmArgs& a, const PackedB& w) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(a.A) | reinterpret_cast<uintptr_t>(a.C) | reinterpret_cast<uintptr_t>(a.pre) |
                       reinterpret_cast<uintptr_t>(a.res);
  return w.main && st.gave_up && tensor_state().ok && !(at & 15) && a.lda % 4 == 0 && a.ldc % 4 == 0 && a.ldp % 4 == 0 && a.ldr % 4 == 0;
}

// One GEMM or two (of one epilogue and format, neither of which reads what the other writes).
void gemm_tensor(Stream& st, Arena& arena, const GemmTask* given, int n) {
  GemmTask q[2];
  const Arena::Mark mark = arena.mark();
  for (int i = 0; i < n; ++i) {
    q[i] = given[i];
    if (!scales_rows(q[i].w.fmt) || q[i].a.a_max) continue;
    uint32_t* mx = arena.alloc<uint32_t>(q[i].a.M);
    row_max(st, mx, q[i].a.A, q[i].a.lda, q[i].a.M, q[i].a.K);
    q[i].a.a_max = mx;
  }
  switch (q[0].a.epi) {
    case EPI_PLAIN: run_tensor<EPI_PLAIN>(st, q, n); break;
    case EPI_SILU: run_tensor<EPI_SILU>(st, q, n); break;
    case EPI_SWIGLU: run_tensor<EPI_SWIGLU>(st, q, n); break;
    case EPI_SILU_BWD: run_tensor<EPI_SILU_BWD>(st, q, n); break;
    case EPI_SWIGLU_BWD: run_tensor<EPI_SWIGLU_BWD>(st, q, n); break;
    case EPI_COMPRESS: run_tensor<EPI_COMPRESS>(st, q, n); break;
    default: throw Error(3, "gemm: unknown epilogue");
  }
  arena.rewind(mark);
}

void gemm_tensor_error_ask(Stream& st, int* host) {
  *host = 0;
  cudaMemcpyAsync(host, st.gave_up, sizeof(int), cudaMemcpyDeviceToHost, st.s);
}
bool gemm_tensor_error(Stream& st, const int* host) {
  if (*host) cudaMemsetAsync(st.gave_up, 0, sizeof(int), st.s);
  return *host != 0;
}

}  // namespace petb
