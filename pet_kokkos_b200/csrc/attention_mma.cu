// The attention's forward on tf32 instructions: warp-level mma.sync m16n8k8 with fp32 accumulation, in two forms. X3 (the
// reference's AttentionMode::TF32x3, src/attention.cpp:949-1011): every operand split into a leading tf32 part and
// its remainder, three products per tile, small terms first. Single pass (AttentionMode::TF32,
// src/attention.cpp:1031-1225 with X3 = false): operands rounded to tf32, one product per tile. Same mathematics as
// attention.cu. attention_f16.cu is faster; this forward serves the models whose energies depend on its bits (AttnArgs::tf32).
//
// One CTA per (atom, head), one warp per block of 16 query rows. The head's Q, K, V slices are staged once with a pitch
// of head_dim + 4 floats, which makes every fragment load below conflict-free:
//   X^T as B operand (scores Q K^T): b(k = t, n = g) = X[key 8kb + g][k0 + t]   -> banks 4g + t
//   X as B operand (P V): the eight contraction indices of a step are taken in the order 0,2,4,6,1,3,5,7, so
//   b(k = t) = X[8kb + 2t][d0 + g], b(k = t + 4) = X[8kb + 2t + 1][d0 + g]
//   -> banks 8t + g; with that order the accumulator fragment of the scores (c0, c1 hold columns
//   2t, 2t + 1) IS the A fragment of the next product, so probabilities never leave registers.
// All scores of a query block stay in registers for the row max and sum. Every sum has one owner and a fixed order.
#include <cstdlib>

#include "attention.h"

namespace petb {

namespace {

constexpr float kOff = -1e30f;
__device__ __forceinline__ bool is_off(float lc) { return lc < -1e29f; }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// The largest magnitude of one row's values, held by the four lanes of a quad as KS pairs (c0, c1) of an accumulator,
// raised into mx[row] (the GEMM that reads the rows scales them by it).
template <int KS>
__device__ __forceinline__ void raise_row(uint32_t* mx, size_t row, bool live, const float (*acc)[4], int c, float scale, int t) {
  float m = 0.f;
#pragma unroll
  for (int db = 0; db < KS; ++db) m = fmaxf(m, fmaxf(fabsf(acc[db][c] * scale), fabsf(acc[db][c + 1] * scale)));
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1)), m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
  if (live && t == 0) atomicMax(mx + row, __float_as_uint(m));
}

struct Frag {
  uint32_t hi, lo;
};
// x = hi + lo with hi the leading 11 significant bits of x (truncated) and lo the remainder rounded to 11 bits
// (half of the last kept bit added, then masked). Integer and fp32-add instructions only: cvt.rna.tf32 runs on the
// quarter-rate conversion pipe, which two conversions per operand element had saturated.
// Single pass (X3 false): hi is x rounded to tf32 (nearest, half of the last kept bit added before the mask) and lo is
// never read, so the compiler drops it.
template <bool X3>
__device__ __forceinline__ Frag split(float x) {
  Frag f;
  if (X3) {
    f.hi = __float_as_uint(x) & 0xFFFFE000u;
    f.lo = (__float_as_uint(x - __uint_as_float(f.hi)) + 0x1000u) & 0xFFFFE000u;
  } else {
    f.hi = (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u;
    f.lo = 0u;
  }
  return f;
}
__device__ __forceinline__ void mma(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The same for G independent accumulators that share the A operand, one term at a time: consecutive
// instructions never depend on each other, so the tensor pipe's latency is covered inside one warp.
template <int G, bool X3>
__device__ __forceinline__ void mma3_shared_a(float (*c)[4], const Frag* a, const Frag (*b)[2]) {
  if (X3) {
#pragma unroll
    for (int j = 0; j < G; ++j) mma(c[j], a[0].lo, a[1].lo, a[2].lo, a[3].lo, b[j][0].hi, b[j][1].hi);
#pragma unroll
    for (int j = 0; j < G; ++j) mma(c[j], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[j][0].lo, b[j][1].lo);
  }
#pragma unroll
  for (int j = 0; j < G; ++j) mma(c[j], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[j][0].hi, b[j][1].hi);
}
__host__ __device__ inline int round16(int s) { return (s + 15) / 16 * 16; }
// Asynchronous 16-byte copies global -> shared: every tile's loads are in flight together, and no register waits on
// them; stage_wait() before the barrier that publishes the tiles.
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

template <int HD>
__device__ __forceinline__ void stage(float* dst, const float* src, size_t ld, int col, int n, int N, int e0, int cnt, int rows) {
  constexpr int Q = HD / 4, P = HD + 4;
  for (int t = threadIdx.x; t < rows * Q; t += blockDim.x) {
    const int r = t / Q, c = (t % Q) * 4;
    if (r < cnt) {
      const size_t row = r == 0 ? size_t(n) : size_t(N) + e0 + r - 1;
      cp_async16(dst + r * P + c, src + row * ld + col + c);
    } else {
      *reinterpret_cast<float4*>(dst + r * P + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// The A fragments (hi, lo) of rows r0.. r0+15 of X [.][P] for every 8-wide step of the head dimension.
template <int HD, bool X3>
__device__ __forceinline__ void load_a(Frag (*f)[4], const float* x, int r0, int g, int t) {
  constexpr int P = HD + 4;
#pragma unroll
  for (int ks = 0; ks < HD / 8; ++ks) {
    f[ks][0] = split<X3>(x[(r0 + g) * P + 8 * ks + t]);
    f[ks][1] = split<X3>(x[(r0 + g + 8) * P + 8 * ks + t]);
    f[ks][2] = split<X3>(x[(r0 + g) * P + 8 * ks + t + 4]);
    f[ks][3] = split<X3>(x[(r0 + g + 8) * P + 8 * ks + t + 4]);
  }
}

template <int HD, int MAXKB, bool X3>
__global__ void __launch_bounds__(32 * ((MAXKB + 1) / 2), MAXKB <= 10 ? 4 : 1) k_attn_fwd_mma(AttnArgs p) {
  after_previous();
  constexpr int P = HD + 4, KS = HD / 8, R = 8 * MAXKB;  // R: staged token rows, the kernel's most (zero past the atom's)
  constexpr int G = MAXKB % 5 == 0 ? 5 : (MAXKB % 4 == 0 ? 4 : 2);  // key blocks whose score tiles advance together
  extern __shared__ __align__(16) float smem[];
  const int n = blockIdx.x / p.H, h = blockIdx.x % p.H, D = p.H * HD;
  const int e0 = p.off[n], cnt = p.off[n + 1] - e0 + 1;
  // key blocks of 8 that hold a token at all: a block past them is zero rows with their cutoff off, and adds nothing
  const int S16 = round16(cnt), nkb = (cnt + 7) / 8;
  float* sq = smem;
  float* sk = sq + R * P;
  float* sv = sk + R * P;
  float* slc = sv + R * P;
  stage<HD>(sq, p.qkv, 3 * size_t(D), h * HD, n, p.N, e0, cnt, S16);
  stage<HD>(sk, p.qkv, 3 * size_t(D), D + h * HD, n, p.N, e0, cnt, R);
  stage<HD>(sv, p.qkv, 3 * size_t(D), 2 * D + h * HD, n, p.N, e0, cnt, R);
  for (int r = threadIdx.x; r < R; r += blockDim.x) {
    const float cf = r == 0 ? 1.0f : (r < cnt ? p.cut[e0 + r - 1] : 0.f);
    slc[r] = cf > 0.f ? __logf(cf) : kOff;
  }
  stage_wait();
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = 16 * warp;
  if (r0 >= cnt) return;

  Frag qf[KS][4];
  load_a<HD, X3>(qf, sq, r0, g, t);
  float s[MAXKB][4];
#pragma unroll
  for (int kb = 0; kb < MAXKB; ++kb) s[kb][0] = s[kb][1] = s[kb][2] = s[kb][3] = 0.f;
#pragma unroll
  for (int kg = 0; kg < MAXKB; kg += G) {
    if (kg < nkb) {  // the same for the whole CTA; a group's blocks past the atom's keys read zero rows
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        Frag b[G][2];
#pragma unroll
        for (int j = 0; j < G; ++j) {
          b[j][0] = split<X3>(sk[(8 * (kg + j) + g) * P + 8 * ks + t]);
          b[j][1] = split<X3>(sk[(8 * (kg + j) + g) * P + 8 * ks + t + 4]);
        }
        mma3_shared_a<G, X3>(&s[kg], qf[ks], b);
      }
    }
  }
  // bias, row max, exponentials, row sum; this lane holds rows g and g + 8, keys 8kb + 2t and + 1
  float m0 = kOff, m1 = kOff;
#pragma unroll
  for (int kb = 0; kb < MAXKB; ++kb)
    if (kb < nkb) {
      const float lc0 = slc[8 * kb + 2 * t], lc1 = slc[8 * kb + 2 * t + 1];
      s[kb][0] = is_off(lc0) ? kOff : s[kb][0] * p.sc + lc0;
      s[kb][1] = is_off(lc1) ? kOff : s[kb][1] * p.sc + lc1;
      s[kb][2] = is_off(lc0) ? kOff : s[kb][2] * p.sc + lc0;
      s[kb][3] = is_off(lc1) ? kOff : s[kb][3] * p.sc + lc1;
      m0 = fmaxf(m0, fmaxf(s[kb][0], s[kb][1]));
      m1 = fmaxf(m1, fmaxf(s[kb][2], s[kb][3]));
    }
  m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 1)), m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 2));
  m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 1)), m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 2));
  float l0 = 0.f, l1 = 0.f;
#pragma unroll
  for (int kb = 0; kb < MAXKB; ++kb)
    if (kb < nkb) {
      s[kb][0] = is_off(s[kb][0]) ? 0.f : __expf(s[kb][0] - m0);
      s[kb][1] = is_off(s[kb][1]) ? 0.f : __expf(s[kb][1] - m0);
      s[kb][2] = is_off(s[kb][2]) ? 0.f : __expf(s[kb][2] - m1);
      s[kb][3] = is_off(s[kb][3]) ? 0.f : __expf(s[kb][3] - m1);
      l0 += s[kb][0] + s[kb][1];
      l1 += s[kb][2] + s[kb][3];
    }
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1), l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1), l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const int q0 = r0 + g, q1 = r0 + g + 8;
  const bool dead0 = q0 > 0 && is_off(slc[q0]), dead1 = q1 > 0 && is_off(slc[q1]);  // a query on an edge at its cutoff
  const float il0 = (!dead0 && l0 > 0.f) ? 1.0f / l0 : 0.f, il1 = (!dead1 && l1 > 0.f) ? 1.0f / l1 : 0.f;

  // O = P V, the probabilities going straight from the accumulator layout into the A operand
  float o[KS][4];
#pragma unroll
  for (int db = 0; db < KS; ++db) o[db][0] = o[db][1] = o[db][2] = o[db][3] = 0.f;
#pragma unroll
  for (int kb = 0; kb < MAXKB; ++kb)
    if (kb < nkb) {
      const Frag a[4] = {split<X3>(s[kb][0] * il0), split<X3>(s[kb][2] * il1), split<X3>(s[kb][1] * il0), split<X3>(s[kb][3] * il1)};
      Frag b[KS][2];
#pragma unroll
      for (int db = 0; db < KS; ++db) {
        b[db][0] = split<X3>(sv[(8 * kb + 2 * t) * P + 8 * db + g]);
        b[db][1] = split<X3>(sv[(8 * kb + 2 * t + 1) * P + 8 * db + g]);
      }
      mma3_shared_a<KS, X3>(o, a, b);
    }
  const size_t g0 = q0 == 0 ? size_t(n) : size_t(p.N) + e0 + q0 - 1, g1 = size_t(p.N) + e0 + q1 - 1;
#pragma unroll
  for (int db = 0; db < KS; ++db) {
    if (q0 < cnt) *reinterpret_cast<float2*>(p.merged + g0 * D + h * HD + 8 * db + 2 * t) = make_float2(o[db][0], o[db][1]);
    if (q1 < cnt) *reinterpret_cast<float2*>(p.merged + g1 * D + h * HD + 8 * db + 2 * t) = make_float2(o[db][2], o[db][3]);
  }
  if (p.merged_max) {
    raise_row<KS>(p.merged_max, g0, q0 < cnt, o, 0, 1.f, t);
    raise_row<KS>(p.merged_max, g1, q1 < cnt, o, 2, 1.f, t);
  }
  if (t == 0 && p.ml) {
    if (q0 < cnt) p.ml[(g0 * p.H + h) * 2] = dead0 ? kOff : m0, p.ml[(g0 * p.H + h) * 2 + 1] = il0;
    if (q1 < cnt) p.ml[(g1 * p.H + h) * 2] = dead1 ? kOff : m1, p.ml[(g1 * p.H + h) * 2 + 1] = il1;
  }
}

bool enabled() {
  static const bool on = [] {
    const char* e = std::getenv("PET_ATTN_MMA");
    return !(e && e[0] == '0');
  }();
  return on;
}

size_t fwd_bytes(int maxkb, int HD) {
  const int R = 8 * maxkb;
  return sizeof(float) * (3 * size_t(R) * (HD + 4) + R);
}
template <class K>
void launch(Stream& st, K kernel, const AttnArgs& p, size_t bytes, int threads, SmemOptIn& opted) {
  opt_in_shared_memory(kernel, bytes, opted);
  launch(st, kernel, p.N * p.H, threads, bytes, p);
  PETB_LAUNCH_CHECK(st);
}

template <int HD, bool X3>
bool fwd_hd(Stream& st, const AttnArgs& p) {
  const int S16 = round16(p.S), threads = 32 * (S16 / 16);
  if (S16 > 176 || fwd_bytes(22, HD) > 200 * 1024) return false;
  static SmemOptIn o10, o16, o22;
  if (S16 <= 80) launch(st, k_attn_fwd_mma<HD, 10, X3>, p, fwd_bytes(10, HD), threads, o10);
  else if (S16 <= 128) launch(st, k_attn_fwd_mma<HD, 16, X3>, p, fwd_bytes(16, HD), threads, o16);
  else launch(st, k_attn_fwd_mma<HD, 22, X3>, p, fwd_bytes(22, HD), threads, o22);
  return true;
}
template <bool X3>
bool fwd_any(Stream& st, const AttnArgs& p) {
  switch (p.hd) {
    case 16: return fwd_hd<16, X3>(st, p);
    case 32: return fwd_hd<32, X3>(st, p);
    case 64: return fwd_hd<64, X3>(st, p);
    default: return false;
  }
}
}  // namespace

// True if the tensor-core kernel took the pass; false leaves it to the other kernels.
bool attention_forward_mma(Stream& st, const AttnArgs& p) {
  if (!enabled()) return false;
  return p.mode == ATTN_TF32 ? fwd_any<false>(st, p) : fwd_any<true>(st, p);
}

}  // namespace petb
