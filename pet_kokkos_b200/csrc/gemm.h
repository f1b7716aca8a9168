// Weight GEMMs with fused epilogues: C[M,N] = A[M,K] . B[N,K]^T (+ bias, residual, activation).
//
// Every dense contraction of the network has a weight as its second operand
// (the reference's weight_gemm, src/ops.cpp:18-24). Weights are held in both
// orientations so that B is always K-major: forward GEMMs read W [N_out, K_in],
// backward (input-adjoint) GEMMs read W^T [K_in, N_out]; no weight gradients are
// formed. The epilogues are the reference's fused ones (src/fused_gemm.cpp:441-563)
// plus the residual add and compress.0's folded geometry/species terms
// (src/ops.cpp:326-365).
//
// Two kernel families:
//   * tensor (gemm_tc.cuh): tcgen05.mma kind::f16 with TMA-fed shared-memory tiles and the accumulator in tensor memory.
//     Operands wider than 16 bits are split into 16-bit parts whose products are summed in fp32; the formats below say
//     into which, for each mode;
//   * fp32 FMA on the CUDA cores (gemm_simt.cu): one accumulation chain per output in k order, the plain product, for callers
//     without a packed weight (pet_gemm_host_static).
// In the native format and on the CUDA cores a row's bits depend on that row and the weight alone, not on how many rows share
// its launch. The other formats add a long K in another order where few rows leave SMs for it (plan_split, gemm_tc.cuh).
#pragma once

#include "common.h"

namespace petb {

enum Epilogue {
  EPI_PLAIN = 0,       // C = acc + bias (+ res for rows >= res_row0)
  EPI_SILU = 1,        // z = acc + bias; pre (optional) = z; C = silu(z)
  EPI_SWIGLU = 2,      // z = acc + bias, columns interleaved (v_j, g_j); pre = z; C[M,N/2] = v * sigmoid(g)
  EPI_SILU_BWD = 3,    // C = acc * silu'(pre)
  EPI_SWIGLU_BWD = 4,  // acc = h_adj [M,N]; C[M,2N]: (acc*sg, acc*v*sg*(1-sg)) from pre [M,2N]
  EPI_COMPRESS = 5     // z = acc + b + tab[sp[row]] + wx . (v, |v|); pre = z; C = silu(z)
};

enum GemmMode { GEMM_NATIVE = 0, GEMM_TF32 = 1, GEMM_BF16 = 2, GEMM_TF32X3 = 3 };

// How an fp32 operand is handed to the 16-bit tensor cores. The fp16 formats scale it by a power of two first: s brings the
// largest value of the row, of A and of B alike, to [2^14, 2^15).
//   FMT_F16X3 (native)   s x = h + m + l: h is s x rounded to a multiple of 2^8, eight bits of the row's largest value; what
//                        remains goes into two fp16 parts. Every value is represented to its last bit, or to 2^-23 of itself
//                        down to 2^-17 of the row's largest; below that to 2^-40 of the largest. Six products; h.h on its own
//                        accumulator, where 1024 columns of K sum without any rounding; the rest (hm mh mm hl lh, 2^-8 of it
//                        and less) on another. The two meet in one fp32 addition. Left out are ml and lm: below 2^-27 of a
//                        product of two values with a leading part, 2^-20 of one where one has none (it lies below 2^-8 of
//                        its row's largest), 2^-12 where neither has.
//   FMT_F16X3_FULL       the same parts, ml and lm among the products. A sum mostly of products without leading parts takes rows
//                        of A and of the weight that are large in different columns (a gain and what undoes it): a weight with
//                        rows or columns like that (k_row_unscale, k_column_spread) runs in this format. Columns that share
//                        factors of 2^-8 .. 2^8 then give an error of 2^-20 of sum |a||w|, with six products 2^-14. What remains
//                        is the second accumulator's truncation, where most of a sum goes over it: what 3xTF32 has. For every
//                        weight it would cost a 1728-atom evaluation 11 % (and a fourth part, x to eleven bits as l's partner,
//                        12 %); as a test in the issuer's loop a small structure's pass 1.5 to 4 %.
//   FMT_F16X2 (3xTF32)   s x = h + l, two fp16 parts: 22 bits or more for every value down to 2^-18 of the row's largest, an
//                        error of 2^-40 of the largest below that. Three products (hl lh hh), one accumulator.
//   FMT_TF32X2 (3xTF32)  x = h + l, two tf32 parts: h is x as the tensor core reads it (its leading 11 bits, truncated), l the
//                        rest rounded to tf32. Three products of 8 columns of K each, one accumulator: twice FMT_F16X2's
//                        operand bytes and twice its instructions.
//   FMT_F16 (tf32)       x's leading 11 bits, truncated: the value a tf32 tensor core reads of x, as one fp16.
//   FMT_TF32 (tf32)      x as it is, read by a tf32 tensor core: the same operand value as FMT_F16's for twice the bytes.
//   FMT_BF16 (bf16)      x rounded to bf16.
enum Format { FMT_F16X3 = 0, FMT_F16X2 = 1, FMT_F16 = 2, FMT_BF16 = 3, FMT_TF32X2 = 4, FMT_TF32 = 5, FMT_F16X3_FULL = 6 };
inline Format format_of(int mode) {
  return mode == GEMM_TF32X3 ? FMT_F16X2 : mode == GEMM_TF32 ? FMT_F16 : mode == GEMM_BF16 ? FMT_BF16 : FMT_F16X3;
}
constexpr bool three_parts(int fmt) { return fmt == FMT_F16X3 || fmt == FMT_F16X3_FULL; }
constexpr bool scales_rows(int fmt) { return three_parts(fmt) || fmt == FMT_F16X2 || fmt == FMT_F16; }

// A weight [rows, K] in one format, made once when it was loaded. K is padded with zeros to a multiple of 32.
//   FMT_F16X3   main [rows][Kp/32][h 32 | m 32], low [rows][Kp] the l parts; `unscale` [rows] what undoes each row's scale, a power
//               of two as bf16, with zeros up to a multiple of eight; behind them a word: whether the values are spread
//   FMT_F16X2   main [rows][Kp/32][h 32 | l 32]; `unscale`
//   FMT_F16     main [rows][Kp]; `unscale`
//   FMT_BF16    main [rows][Kp]
//   FMT_TF32X2  main [rows][Kp] and low [rows][Kp], fp32 words; FMT_TF32 main alone
struct PackedB {
  Format fmt = FMT_F16X3;
  const uint16_t* main = nullptr;
  const uint16_t* low = nullptr;
  const uint16_t* unscale = nullptr;
  int Kp = 0;
};
inline int packed_k(int K) { return (K + 31) / 32 * 32; }
constexpr size_t unscale_halves(int rows) { return size_t(rows + 7) / 8 * 8 + 8; }
// 16-bit values and bytes a packed weight takes (main and low together), rows padded apart to 16 bytes.
inline size_t packed_halves(int fmt, int rows, int K) {
  return size_t(rows) * packed_k(K) * (three_parts(fmt) ? 3 : fmt == FMT_F16X2 || fmt == FMT_TF32 ? 2 : fmt == FMT_TF32X2 ? 4 : 1);
}
// Packs W [rows, K] (element (r, k) at W[r * ld_r + k * ld_k]) into `out`, and writes `unscale` (unscale_halves(rows),
// 16-byte aligned).
PackedB pack_weight(cudaStream_t s, Format fmt, const float* W, size_t ld_r, size_t ld_k, int rows, int K, uint16_t* out, uint16_t* unscale);
// Whether pack_weight found the values of a weight in FMT_F16X3 spread. Copies a word from the device: the packing has to have ended.
bool values_spread(const PackedB& w, int rows);
// Such a weight becomes one in FMT_F16X3_FULL.
void full_if_spread(PackedB& w, int rows);

struct GemmArgs {
  const float* A = nullptr;  // [M,K]
  int lda = 0;
  const float* B = nullptr;  // [N,K] fp32: read by the CUDA-core kernel alone
  int ldb = 0;
  PackedB nat, fast;         // B in the native format, and in the one this GEMM runs in
  // The fp16 formats scale each row of A: the bits of the row's largest |value| (0 for a row of zeros),
  // kept up to date by whatever wrote A. Null: found by a pass over A.
  const uint32_t* a_max = nullptr;
  // Unless null, each row's largest |C| is raised into c_max (atomicMax on the bits; the caller zeroed it).
  uint32_t* c_max = nullptr;
  // EPI_PLAIN, EPI_SWIGLU in the formats of several parts: the product of A's rows over their root mean squares (an RMSNorm, its
  // gain in the weight), unless 0; to the kernel 1 / K.
  float rms = 0.f;
  float* C = nullptr;        // [M, N] (EPI_SWIGLU: [M,N/2]; EPI_SWIGLU_BWD: [M,2N])
  int ldc = 0;
  int M = 0, N = 0, K = 0;
  const float* bias = nullptr;  // [N]
  const float* res = nullptr;   // [M,N] residual, read before C is written (may alias C)
  int ldr = 0;
  int res_row0 = 0;
  float* pre = nullptr;  // saved or read pre-activation
  int ldp = 0;
  // EPI_COMPRESS
  const float* tab = nullptr;    // [n_species, N]
  const int* sp = nullptr;       // [M]
  const float* wx = nullptr;     // [N,4]
  const double* vec = nullptr;   // [M,3]
  const double* dist = nullptr;  // [M]
  int epi = EPI_PLAIN;
};

// Runs the GEMM in the format of `fast`, or of `nat` where it has fewer than 64 rows.
void gemm(Stream& st, Arena& arena, const GemmArgs& a);
// Two that do not depend on each other and share no output, as one launch where that is the faster way (plan_two, gemm_tc.cuh);
// `a` the one of fewer rows and longer contraction.
void gemm_two(Stream& st, Arena& arena, const GemmArgs& a, const GemmArgs& b);

// out[M] = A[M,K] . w[K] + b (a one-column linear layer), one warp per row.
void gemv_rows(Stream& st, const float* A, int lda, const float* w, const float* bias, float* out, int M, int K);

// mx[r] = bits of the largest |x(r, :)|.
void row_max(Stream& st, uint32_t* mx, const float* x, int ld, int R, int D);

// Whether a tensor-core kernel of this stream gave up on a bounded wait: the first puts a copy of the stream's word into pinned
// memory, the second, once the stream has got there, looks at it and clears the word.
void gemm_tensor_error_ask(Stream& st, int* host);
bool gemm_tensor_error(Stream& st, const int* host);

// True once the tensor-core path has been initialised on this device (driver entry point found).
bool tensor_gemm_available();

}  // namespace petb
