// The fp32 GEMM on the CUDA cores and the GEMM dispatcher: see gemm.h.
//
// 128 x 128 x 16 tiles, 256 threads, 8 x 8 outputs per thread, operands staged in
// shared memory (transposed, so the inner loop reads float4s) with the next tile's
// global loads issued before the current tile's arithmetic. Each output is one
// chain of fused multiply-adds over k in increasing order, whatever the tile or
// the row count: a row's result depends on that row alone. It serves callers whose
// weight has no packed form (pet_gemm_host_static): with the weight's parts at hand
// the tensor cores are four times faster and no less exact.
#include "epilogue.cuh"
#include "gemm_tc.h"

namespace petb {

void gemm_tensor(Stream& st, Arena& arena, const GemmTask* q, int n);  // gemm_tc.cu
bool gemm_tensor_usable(const Stream& st, const GemmArgs& a, const PackedB& w);

namespace {

constexpr int BM = 128, BN = 128, BK = 16, PAD = 4;

// Two fp32 values in one 64-bit register, and the packed fused multiply-add of sm_100: d.x = a.x * b.x + d.x and
// d.y = a.y * b.y + d.y, each rounded once (round to nearest even), as fmaf does.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__global__ void __launch_bounds__(256, 2) k_gemm_native(GemmArgs p) {
  after_previous();
  __shared__ __align__(16) float As[2][BK][BM + PAD];
  __shared__ __align__(16) float Bs[2][BK][BN + PAD];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int tiles_n = (p.N + BN - 1) / BN;
  const int m0 = (blockIdx.x / tiles_n) * BM, n0 = (blockIdx.x % tiles_n) * BN;

  // Loader: a thread brings rows lr and lr + 64 of each tile, four k values at lk.
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  float4 ra[2], rb[2];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int am = m0 + lr + 64 * h, bn = n0 + lr + 64 * h, k = k0 + lk;
      ra[h] = (am < p.M && k < p.K) ? ld4(p.A + size_t(am) * p.lda + k) : make_float4(0, 0, 0, 0);
      rb[h] = (bn < p.N && k < p.K) ? ld4(p.B + size_t(bn) * p.ldb + k) : make_float4(0, 0, 0, 0);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lr + 64 * h;
      As[buf][lk + 0][r] = ra[h].x, As[buf][lk + 1][r] = ra[h].y, As[buf][lk + 2][r] = ra[h].z, As[buf][lk + 3][r] = ra[h].w;
      Bs[buf][lk + 0][r] = rb[h].x, Bs[buf][lk + 1][r] = rb[h].y, Bs[buf][lk + 2][r] = rb[h].z, Bs[buf][lk + 3][r] = rb[h].w;
    }
  };

  // The accumulators as pairs of neighbouring columns: one fma.rn.f32x2 advances two of them with the IEEE fp32
  // fused multiply-add of the scalar instruction (same bits), for half the issue slots.
  unsigned long long acc2[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc2[i][j] = 0ull;

  fetch(0);
  stash(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < p.K; k0 += BK) {
    const bool more = k0 + BK < p.K;
    if (more) fetch(k0 + BK);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float4 a0 = ld4(&As[buf][k][ty * 4]), a1 = ld4(&As[buf][k][64 + ty * 4]);
      const float4 b0 = ld4(&Bs[buf][k][tx * 4]), b1 = ld4(&Bs[buf][k][64 + tx * 4]);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const unsigned long long b2[4] = {pack2(b0.x, b0.y), pack2(b0.z, b0.w), pack2(b1.x, b1.y), pack2(b1.z, b1.w)};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned long long aa = pack2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) fma2(acc2[i][j], aa, b2[j]);
      }
    }
    if (more) {
      stash(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }

  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) unpack2(acc2[i][j], acc[i][2 * j], acc[i][2 * j + 1]);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
    if (row >= p.M) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = n0 + 64 * h + tx * 4;
      if (col < p.N) st4(p.C + size_t(row) * p.ldc + col, ld4(&acc[i][4 * h]));
    }
  }
}

__global__ void k_gemv_rows(const float* __restrict__ A, int lda, const float* __restrict__ w, const float* __restrict__ bias,
                            float* __restrict__ out, int M, int K) {
  after_previous();
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= M) return;
  float s = 0.0f;
  for (int k = lane; k < K; k += 32) s = fmaf(A[size_t(r) * lda + k], w[k], s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[r] = s + (bias ? bias[0] : 0.0f);
}

}  // namespace

namespace {

void check(const GemmArgs& a) {
  if (a.N % 4 || a.K % 4 || a.lda % 4 || (a.B && a.ldb % 4) || a.ldc % 2)
    throw Error(2, "gemm: widths must be multiples of 4 (N=" + std::to_string(a.N) + ", K=" + std::to_string(a.K) + ")");
}
// Algorithmic work: 2MNK flops; A, B, C once each, plus what the epilogue reads and writes.
double flops_of(const GemmArgs& a) { return 2.0 * a.M * a.N * a.K; }
double bytes_of(const GemmArgs& a) {
  double bytes = 4.0 * (double(a.M) * a.K + double(a.N) * a.K + double(a.M) * a.N);
  if (a.res) bytes += 4.0 * a.M * a.N;
  if (a.pre) bytes += 4.0 * a.M * a.N * (a.epi == EPI_SWIGLU_BWD ? 2.0 : 1.0);
  if (a.epi == EPI_SWIGLU) bytes -= 2.0 * a.M * a.N;      // h is half as wide as the product
  if (a.epi == EPI_SWIGLU_BWD) bytes += 4.0 * a.M * a.N;  // pre_adj is twice as wide
  return bytes;
}
// Fewer than half a tile of rows: the speed modes' products would not be felt there, so they run at full precision.
const PackedB& weight_of(const GemmArgs& a) { return a.M < 64 || a.N < 32 ? a.nat : a.fast; }

}  // namespace

void gemm(Stream& st, Arena& arena, const GemmArgs& a) {
  if (a.M <= 0 || a.N <= 0) return;
  check(a);
  const ProfScope ps(st, PC_GEMM, flops_of(a), bytes_of(a));
  const GemmTask q{a, weight_of(a)};
  if (gemm_tensor_usable(st, a, q.w)) return gemm_tensor(st, arena, &q, 1);
  if (!a.B) throw Error(3, "gemm: this weight has no fp32 copy for the CUDA cores");
  if (a.epi != EPI_PLAIN || a.bias || a.res || a.c_max || a.rms != 0.f) throw Error(3, "gemm: the CUDA cores give the plain product alone");
  const long long tiles = (long long) cdiv(a.M, BM) * cdiv(a.N, BN);
  launch(st, k_gemm_native, (unsigned) tiles, 256, 0, a);
  PETB_LAUNCH_CHECK(st);
}

void gemm_two(Stream& st, Arena& arena, const GemmArgs& a, const GemmArgs& b) {
  const bool one_launch = a.M > 0 && b.M > 0 && a.N > 0 && b.N > 0 && a.epi == b.epi && weight_of(a).fmt == weight_of(b).fmt &&
                          gemm_tensor_usable(st, a, weight_of(a)) && gemm_tensor_usable(st, b, weight_of(b));
  if (!one_launch) {
    gemm(st, arena, a);
    return gemm(st, arena, b);
  }
  check(a), check(b);
  const ProfScope ps(st, PC_GEMM, flops_of(a) + flops_of(b), bytes_of(a) + bytes_of(b));
  const GemmTask q[2] = {{a, weight_of(a)}, {b, weight_of(b)}};
  gemm_tensor(st, arena, q, 2);
}

void gemv_rows(Stream& st, const float* A, int lda, const float* w, const float* bias, float* out, int M, int K) {
  if (M <= 0) return;
  const ProfScope ps(st, PC_GEMM, 2.0 * M * K, 4.0 * (double(M) * K + K + M));
  launch(st, k_gemv_rows, cdiv((long long) M * 32, 256), 256, 0, A, lda, w, bias, out, M, K);
  PETB_LAUNCH_CHECK(st);
}

}  // namespace petb
