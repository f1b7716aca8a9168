// Attention on the tensor cores: warp-level mma.sync m16n8k16 on fp16 parts with fp32 accumulation. Same mathematics as
// attention.cu; used when an atom's tokens fit shared memory.
//
// An operand is scaled by a power of two that brings its largest value (of this atom and head, found while the tile is staged: Q, K,
// V and dO each have their own, whatever the other heads hold) to [2^14, 2^15) and split into P parts:
//   P = 3 (ATTN_NATIVE)  x = h + m + l, h a multiple of 2^8: eight bits of the largest value, so that the h.h products of up to
//                        1024 terms sum exactly; six products, h.h on an accumulator of its own (gemm.h has the argument): hh hm
//                        mh mm tl lt with t = h + m to eleven bits, added up in registers. With h for t, as the GEMMs do on
//                        weights that are not spread, ml and lm are left out; scores whose queries and keys are large in
//                        different columns then put a force 1.7e-5 of the scale off for 2e-6. What an atom holds is not known
//                        ahead, so the tile always takes t: attention of diamond1728 1.20 + 3.25 ms -> 1.32 + 3.44 (ml and lm as
//                        products of their own: 1.38 + 3.85);
//   P = 2 (ATTN_TF32X3)  x = h + l, 22 bits; three products;
//   P = 1 (ATTN_TF32)    x rounded to 11 bits; one product.
// Q, K, V (and dO) are split once, when a CTA stages its (atom, head): the parts of a row lie side by side in shared memory,
// rows an odd number of 16-byte slots apart, so that ldmatrix (plain for X^T as B operand, transposed for X) is free
// of conflicts. What a product makes in registers (probabilities, score adjoints) is split there: two 8-column accumulators
// of one product are the A operand of the next.
//
// One CTA per (atom, head), one warp per block of 16 rows. Forward: all scores of a query block stay in registers for the
// row max and sum. Backward, with the saved max and 1/sum: a warp takes 16 queries and forms dQ = sc dS K, then 16 keys
// and works transposed (S^T = K Q^T, dP^T = V dO^T), so that dS^T and P^T come out as A operands for dK = sc dS^T Q and
// dV = P^T dO and each key's column sum of dS is a row sum. Nothing S x S is stored and the warps never wait on each other
// once the tile is staged. Every sum has one owner and a fixed order. Exponents are taken to base 2.
//
// What bounds it: latency (a tile's loads; dependent products of three or six instructions; 15 to 20 warps an SM by registers and shared
// memory). Hence small CTAs, three or four of them on an SM at the usual 80 rows: one stages its tile while the others multiply.
#include <cuda_fp16.h>

#include "attention.h"

namespace petb {

namespace {

constexpr float kOff = -1e30f, kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
__device__ __forceinline__ bool is_off(float lc) { return lc < -1e29f; }
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t) __cvta_generic_to_shared(p); }
__host__ __device__ constexpr int round16(int s) { return (s + 15) / 16 * 16; }
template <int HD, int P>
__host__ __device__ constexpr int pitch() { return P * HD * 2 + 16; }  // bytes of a row

__device__ __forceinline__ float exp2_fast(float x) {  // within 2 ulp; what would be subnormal is zero
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The power of two that brings values up to the one with these bits to at most 2^15, and its inverse.
__device__ __forceinline__ uint32_t scale_exponent(uint32_t max_bits) { return min(max(max_bits >> 23, 15u), 253u); }
__device__ __forceinline__ float scale_of(uint32_t max_bits) { return __uint_as_float((268u - scale_exponent(max_bits)) << 23); }
__device__ __forceinline__ float unscale_of(uint32_t max_bits) { return __uint_as_float((scale_exponent(max_bits) - 14u) << 23); }

__device__ __forceinline__ uint32_t pack(float x, float y) {
  const __half2 v = __floats2half2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack(uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }

// Two neighbouring values, already scaled, into P parts.
template <int P>
__device__ __forceinline__ void split2(float x, float y, uint32_t* part) {
  if (P == 3) {
    constexpr float kGrid = 3221225472.f;  // 1.5 2^31: adding it rounds to a multiple of 2^8
    const float hx = (x + kGrid) - kGrid, hy = (y + kGrid) - kGrid;
    part[0] = pack(hx, hy);
    x -= hx, y -= hy;
    part[1] = pack(x, y);
    const float2 m = unpack(part[1]);
    part[2] = pack(x - m.x, y - m.y);
  } else {
    part[0] = pack(x, y);
    if (P == 2) {
      const float2 h = unpack(part[0]);
      part[1] = pack(x - h.x, y - h.y);
    }
  }
}

__device__ __forceinline__ void ldsm4(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma(float* c, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// N accumulators of 16 x 8 that advance together: `big` takes the leading products, `small` (P = 3) the others.
template <int P, int N>
struct Acc {
  float big[N][4], small[P == 3 ? N : 1][4];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        big[n][i] = 0.f;
        if (P == 3) small[n][i] = 0.f;
      }
  }
  __device__ __forceinline__ float get(int n, int i) const { return P == 3 ? big[n][i] + small[n][i] : big[n][i]; }
};
// The products of parts (i, j) in the order they are added, small terms first. With three parts l's partner is h + m to eleven bits
// (part 3, made in registers).
template <int P>
__device__ __forceinline__ constexpr int products() { return P == 3 ? 6 : P == 2 ? 3 : 1; }
template <int P>
__device__ __forceinline__ constexpr int part_a(int u) {
  constexpr int three[6] = {3, 2, 1, 0, 1, 0}, two[3] = {0, 1, 0};
  return P == 3 ? three[u] : P == 2 ? two[u] : 0;
}
template <int P>
__device__ __forceinline__ constexpr int part_b(int u) {
  constexpr int three[6] = {2, 3, 1, 1, 0, 0}, two[3] = {1, 0, 0};
  return P == 3 ? three[u] : P == 2 ? two[u] : 0;
}
template <int P>
__host__ __device__ constexpr int with_sum() { return P == 3 ? 4 : P; }
// Part 3 of a fragment whose first two parts are x[0] and x[1].
template <int P>
__device__ __forceinline__ void add_sum(uint32_t (*x)[4]) {
  if (P == 3) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 v = __hadd2(*reinterpret_cast<const __half2*>(&x[0][i]), *reinterpret_cast<const __half2*>(&x[1][i]));
      x[3][i] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
}

// Rows r0 .. r0 + 15, columns 16 ks .. + 15 of a staged tensor as A operand, part j.
template <int HD, int P>
__device__ __forceinline__ void load_a(uint32_t* a, uint32_t base, int r0, int ks, int j, int lane) {
  ldsm4(a, base + (r0 + (lane & 15)) * pitch<HD, P>() + j * HD * 2 + ks * 32 + (lane >> 4) * 16);
}
// Rows r0 .. r0 + 15 as columns of a B operand (X^T), contraction over columns 16 ks .. + 15: two 8-wide blocks (b[0..1], b[2..3]).
template <int HD, int P>
__device__ __forceinline__ void load_bt(uint32_t* b, uint32_t base, int r0, int ks, int j, int lane) {
  ldsm4(b, base + (r0 + (lane >> 4) * 8 + (lane & 7)) * pitch<HD, P>() + j * HD * 2 + ks * 32 + ((lane >> 3) & 1) * 16);
}
// Rows r0 .. r0 + 15 as the contraction of a B operand (X), columns 16 d .. + 15: two 8-wide blocks.
template <int HD, int P>
__device__ __forceinline__ void load_b(uint32_t* b, uint32_t base, int r0, int d, int j, int lane) {
  ldsm4_t(b, base + (r0 + ((lane >> 3) & 1) * 8 + (lane & 7)) * pitch<HD, P>() + j * HD * 2 + d * 32 + (lane >> 4) * 16);
}

// Two 16 x 16 blocks of X Y^T that share nothing but their rows' and columns' positions: x1 . y1 and x2 . y2 (their A operands kept
// in registers with KEEP, else loaded step by step).
template <int HD, int P, bool KEEP, bool BOTH>
__device__ __forceinline__ void two_products(Acc<P, 2>& c1, Acc<P, 2>& c2, const uint32_t (*a1)[P][4], const uint32_t (*a2)[P][4], uint32_t xa1,
                                             uint32_t xa2, int ra, uint32_t y1, uint32_t y2, int rb, int lane) {
  c1.zero();
  if (BOTH) c2.zero();
#pragma unroll
  for (int ks = 0; ks < HD / 16; ++ks) {
    constexpr int R = with_sum<P>();
    uint32_t b1[R][4], b2[R][4], t1[R][4], t2[R][4];
#pragma unroll
    for (int j = 0; j < P; ++j) {
      load_bt<HD, P>(b1[j], y1, rb, ks, j, lane);
      if (BOTH) load_bt<HD, P>(b2[j], y2, rb, ks, j, lane);
      if (!KEEP) {
        load_a<HD, P>(t1[j], xa1, ra, ks, j, lane);
        if (BOTH) load_a<HD, P>(t2[j], xa2, ra, ks, j, lane);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          t1[j][i] = a1[ks][j][i];
          if (BOTH) t2[j][i] = a2[ks][j][i];
        }
      }
    }
    add_sum<P>(b1), add_sum<P>(t1);
    if (BOTH) add_sum<P>(b2), add_sum<P>(t2);
#pragma unroll
    for (int u = 0; u < products<P>(); ++u) {
      const int i = part_a<P>(u), j = part_b<P>(u);
      const bool lead = u + 1 == products<P>();
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        mma(P == 3 && !lead ? c1.small[P == 3 ? n : 0] : c1.big[n], t1[i], b1[j] + 2 * n);
        if (BOTH) mma(P == 3 && !lead ? c2.small[P == 3 ? n : 0] : c2.big[n], t2[i], b2[j] + 2 * n);
      }
    }
  }
}
// c[16 x HD] += A . X over 16 rows of X. With three parts the block's products meet in accumulators of their own and go onto c
// rounded to nearest: c takes no second set of registers.
template <int HD, int P>
__device__ __forceinline__ void product_rows(float (*c)[4], const uint32_t (*a)[4], uint32_t x, int r0, int lane) {
#pragma unroll
  for (int d = 0; d < HD / 16; ++d) {
    uint32_t b[with_sum<P>()][4];
#pragma unroll
    for (int j = 0; j < P; ++j) load_b<HD, P>(b[j], x, r0, d, j, lane);
    add_sum<P>(b);
    Acc<3, 2> tmp;
    if (P == 3) tmp.zero();
#pragma unroll
    for (int u = 0; u < products<P>(); ++u) {
      const bool lead = u + 1 == products<P>();
#pragma unroll
      for (int n = 0; n < 2; ++n)
        mma(P == 3 ? (lead ? tmp.big[n] : tmp.small[n]) : c[2 * d + n], a[part_a<P>(u)], b[part_b<P>(u)] + 2 * n);
    }
    if (P == 3) {
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) c[2 * d + n][i] += tmp.get(n, i);
    }
  }
}
template <int HD>
__device__ __forceinline__ void clear(float (*c)[4]) {
#pragma unroll
  for (int d = 0; d < HD / 8; ++d) c[d][0] = c[d][1] = c[d][2] = c[d][3] = 0.f;
}
// The A operand whose rows are this lane's g and g + 8: x[n][0..1] of row g, x[n][2..3] of row g + 8, columns 8 n + 2 t, + 1.
template <int P>
__device__ __forceinline__ void make_a(uint32_t (*a)[4], const float (*x)[4]) {
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t part[P];
      split2<P>(x[n][2 * h], x[n][2 * h + 1], part);
#pragma unroll
      for (int j = 0; j < P; ++j) a[j][2 * n + h] = part[j];
    }
  add_sum<P>(a);
}

// A thread's largest value of a tensor raised into the tile's.
__device__ __forceinline__ void raise_tile(uint32_t* slot, float m) {
  const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if ((threadIdx.x & 31) == 0) atomicMax(slot, most);
}
__device__ __forceinline__ float max_abs(float m, const float4& x) {
  return fmaxf(fmaxf(m, fmaxf(fabsf(x.x), fabsf(x.y))), fmaxf(fabsf(x.z), fabsf(x.w)));
}

// A thread's 16 bytes of row r (a token row of the atom) of a tensor, in parts.
template <int HD, int P>
__device__ __forceinline__ void put(uint8_t* dst, int r, int c, const float4& x, int row_bytes = pitch<HD, P>()) {  // (x scaled)
  uint32_t lo[P], hi[P];
  split2<P>(x.x, x.y, lo), split2<P>(x.z, x.w, hi);
#pragma unroll
  for (int j = 0; j < P; ++j) *reinterpret_cast<uint2*>(dst + r * row_bytes + j * HD * 2 + c * 2) = make_uint2(lo[j], hi[j]);
}
__device__ __forceinline__ float4 get(const float* src, size_t at, bool live) {
  return live ? __ldg(reinterpret_cast<const float4*>(src + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ float4 operator*(const float4& x, float s) { return make_float4(x.x * s, x.y * s, x.z * s, x.w * s); }
__device__ __forceinline__ float dot4(const float4& a, const float4& b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }

// The largest magnitude of one row's values, held by the four lanes of a quad, raised into mx[row].
__device__ __forceinline__ void raise_row(uint32_t* mx, size_t row, bool live, float m, int t) {
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1)), m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
  if (live && t == 0) atomicMax(mx + row, __float_as_uint(m));
}

// c (16 x HD), its row g times f0 and its row g + 8 times f1, to columns col.. of rows g0 and g1 of out.
template <int HD>
__device__ __forceinline__ void write_rows(float* out, size_t ld, int col, size_t g0, size_t g1, bool live0, bool live1, const float (*c)[4],
                                           float f0, float f1, uint32_t* mx, int t) {
  float m0 = 0.f, m1 = 0.f;
#pragma unroll
  for (int d = 0; d < HD / 8; ++d) {
    const float x0 = c[d][0] * f0, x1 = c[d][1] * f0, x2 = c[d][2] * f1, x3 = c[d][3] * f1;
    if (live0) *reinterpret_cast<float2*>(out + g0 * ld + col + 8 * d + 2 * t) = make_float2(x0, x1);
    if (live1) *reinterpret_cast<float2*>(out + g1 * ld + col + 8 * d + 2 * t) = make_float2(x2, x3);
    m0 = fmaxf(m0, fmaxf(fabsf(x0), fabsf(x1))), m1 = fmaxf(m1, fmaxf(fabsf(x2), fabsf(x3)));
  }
  if (mx) raise_row(mx, g0, live0, m0, t), raise_row(mx, g1, live1, m1, t);
}

// CTAs of `rows` rows that an SM's shared memory holds, at most four: what their registers are cut for.
template <int HD, int P, int TENSORS>
__host__ __device__ constexpr int resident(int rows) {
  const int n = 220 * 1024 / (rows * (TENSORS * pitch<HD, P>() + 20) + 1024);
  return n > 4 ? 4 : n < 1 ? 1 : n;
}

template <int HD, int P, int MAXB>
__global__ void __launch_bounds__(32 * MAXB, MAXB <= 5 ? resident<HD, P, 3>(16 * MAXB) : 1) k_attn_fwd_f16(AttnArgs p) {
  after_previous();
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ uint32_t s_max[3];  // of Q, K, V
  const int n = blockIdx.x / p.H, h = blockIdx.x % p.H, D = p.H * HD;
  const int e0 = p.off[n], cnt = p.off[n + 1] - e0 + 1;
  const int S16 = round16(cnt), nb = S16 / 16, SM = round16(p.S);
  uint8_t *sq = smem, *sk = sq + SM * pitch<HD, P>(), *sv = sk + SM * pitch<HD, P>();
  float* slc = reinterpret_cast<float*>(sv + SM * pitch<HD, P>());
  // Staging: a thread's loads of U rows' pieces are under way while it sees to the cutoffs; then it looks for the tile's largest
  // values, also among the pieces it takes later (a head size of 64: read here, and again for the split).
  constexpr int Q = HD / 4, U = 4;
  float4 x0[U], x1[U], x2[U];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * blockDim.x, r = t / Q;
      const size_t at = (r == 0 ? size_t(n) : size_t(p.N) + e0 + r - 1) * 3 * D + h * HD + (t % Q) * 4;
      x0[u] = get(p.qkv, at, r < cnt), x1[u] = get(p.qkv, at + D, r < cnt), x2[u] = get(p.qkv, at + 2 * D, r < cnt);
    }
  };
  fetch(threadIdx.x);
  if (threadIdx.x < 3) s_max[threadIdx.x] = 0;
  for (int r = threadIdx.x; r < S16; r += blockDim.x) {
    const float cf = r == 0 ? 1.0f : (r < cnt ? p.cut[e0 + r - 1] : 0.f);
    slc[r] = cf > 0.f ? __logf(cf) * kLog2e : kOff;
  }
  __syncthreads();
  {
    float mq = 0.f, mk = 0.f, mv = 0.f;
    for (int t = threadIdx.x + U * blockDim.x; t < cnt * Q; t += blockDim.x) {
      const int r = t / Q;
      const size_t at = (r == 0 ? size_t(n) : size_t(p.N) + e0 + r - 1) * 3 * D + h * HD + (t % Q) * 4;
      mq = max_abs(mq, get(p.qkv, at, true)), mk = max_abs(mk, get(p.qkv, at + D, true)), mv = max_abs(mv, get(p.qkv, at + 2 * D, true));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) mq = max_abs(mq, x0[u]), mk = max_abs(mk, x1[u]), mv = max_abs(mv, x2[u]);
    raise_tile(s_max, mq), raise_tile(s_max + 1, mk), raise_tile(s_max + 2, mv);
  }
  __syncthreads();
  const float scq = scale_of(s_max[0]), sck = scale_of(s_max[1]), scv = scale_of(s_max[2]);
  for (int t0 = threadIdx.x; t0 < S16 * Q; t0 += U * blockDim.x) {
    if (t0 != threadIdx.x) fetch(t0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * blockDim.x, r = t / Q, c = (t % Q) * 4;
      if (t >= S16 * Q) break;
      put<HD, P>(sq, r, c, x0[u] * scq), put<HD, P>(sk, r, c, x1[u] * sck), put<HD, P>(sv, r, c, x2[u] * scv);
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = 16 * warp;
  if (r0 >= cnt) return;
  const uint32_t aq = smem_u32(sq), ak = smem_u32(sk), av = smem_u32(sv);
  const float us = unscale_of(s_max[2]), f = unscale_of(s_max[0]) * unscale_of(s_max[1]) * p.sc * kLog2e;
  uint32_t qa[HD / 16][P][4];
#pragma unroll
  for (int ks = 0; ks < HD / 16; ++ks)
#pragma unroll
    for (int j = 0; j < P; ++j) load_a<HD, P>(qa[ks][j], aq, r0, ks, j, lane);
  float x[MAXB][2][4];
  float m0 = kOff, m1 = kOff;
#pragma unroll
  for (int b = 0; b < MAXB; ++b)
    if (b < nb) {
      Acc<P, 2> c, none;
      two_products<HD, P, true, false>(c, none, qa, qa, aq, aq, r0, ak, ak, 16 * b, lane);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float l0 = slc[16 * b + 8 * i + 2 * t], l1 = slc[16 * b + 8 * i + 2 * t + 1];
        x[b][i][0] = fmaf(c.get(i, 0), f, l0), x[b][i][1] = fmaf(c.get(i, 1), f, l1);
        x[b][i][2] = fmaf(c.get(i, 2), f, l0), x[b][i][3] = fmaf(c.get(i, 3), f, l1);
        m0 = fmaxf(m0, fmaxf(x[b][i][0], x[b][i][1]));
        m1 = fmaxf(m1, fmaxf(x[b][i][2], x[b][i][3]));
      }
    }
  m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 1)), m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 2));
  m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 1)), m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 2));
  const float n0 = m0 * kLn2, n1 = m1 * kLn2;  // the maxima as they are saved, and back as the backward will have them
  m0 = n0 * kLog2e, m1 = n1 * kLog2e;
  float l0 = 0.f, l1 = 0.f;
#pragma unroll
  for (int b = 0; b < MAXB; ++b)
    if (b < nb) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {  // a key that is off lies 1e30 below the atom's own token: exp gives its zero
        x[b][i][0] = exp2_fast(x[b][i][0] - m0), x[b][i][1] = exp2_fast(x[b][i][1] - m0);
        x[b][i][2] = exp2_fast(x[b][i][2] - m1), x[b][i][3] = exp2_fast(x[b][i][3] - m1);
        l0 += x[b][i][0] + x[b][i][1];
        l1 += x[b][i][2] + x[b][i][3];
      }
    }
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1), l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1), l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const int q0 = r0 + g, q1 = r0 + g + 8;
  const bool dead0 = q0 > 0 && is_off(slc[q0]), dead1 = is_off(slc[q1]);  // a query on an edge at its cutoff
  const float il0 = (!dead0 && l0 > 0.f) ? 1.0f / l0 : 0.f, il1 = (!dead1 && l1 > 0.f) ? 1.0f / l1 : 0.f;
  const float w0 = il0 * 32768.f, w1 = il1 * 32768.f;  // probabilities are scaled by 2^15
  float o[HD / 8][4];
  clear<HD>(o);
#pragma unroll
  for (int b = 0; b < MAXB; ++b)
    if (b < nb) {
#pragma unroll
      for (int i = 0; i < 2; ++i) x[b][i][0] *= w0, x[b][i][1] *= w0, x[b][i][2] *= w1, x[b][i][3] *= w1;
      uint32_t a[with_sum<P>()][4];
      make_a<P>(a, x[b]);
      product_rows<HD, P>(o, a, av, 16 * b, lane);
    }
  const size_t g0 = q0 == 0 ? size_t(n) : size_t(p.N) + e0 + q0 - 1, g1 = size_t(p.N) + e0 + q1 - 1;
  write_rows<HD>(p.merged, D, h * HD, g0, g1, q0 < cnt, q1 < cnt, o, us * (1.f / 32768.f), us * (1.f / 32768.f), p.merged_max, t);
  if (t == 0 && p.ml) {
    if (q0 < cnt) p.ml[(g0 * p.H + h) * 2] = dead0 ? kOff : n0, p.ml[(g0 * p.H + h) * 2 + 1] = il0;
    if (q1 < cnt) p.ml[(g1 * p.H + h) * 2] = dead1 ? kOff : n1, p.ml[(g1 * p.H + h) * 2 + 1] = il1;
  }
}

// Bytes of a row of V's tile where dS takes its place (ONCE): P parts of as many queries as the tile has rows.
template <int HD, int P>
__host__ __device__ constexpr int shared_pitch(int rows) {
  return pitch<HD, P>() > P * rows * 2 + 16 ? pitch<HD, P>() : P * rows * 2 + 16;
}

// ONCE: a warp per block of 16 keys, no more. Scores and score adjoints are made once, transposed, by the warp that has the keys:
// it sums dK and dV and leaves dS^T, in parts, in the rows of V's tile that are its keys' (nobody else reads those, and it has them
// in registers); then, all warps' dS there, it takes the queries of the same rows for dQ = sc dS K. A query's row of dS^T is left on the
// scale of its own largest value: on the tile's, a row of dO 2^-16 of the largest had 13 bits of dQ left instead of 23
// (one part: 2^-24, four instead of 11). Per 16 x 16 block 60 products instead of 84 (P = 2), 22 ldmatrix instead of 44, half the
// exponentials; V's rows are longer, so fewer CTAs share an SM.
// That alone gave 5 % (P = 1, 2; P = 3 lost 5): the warps waited for the tile's loads (two of eight stalled cycles) and for one another
// behind them. With all of a thread's rows asked for at once (U) instead of in three trips: diamond1728 P = 2 2.16 ms -> 1.87, P = 3 3.64 ->
// 3.57, 16-thousand-atom batch 9.25 -> 8.6, water1791 P = 1 0.737 -> 0.705 (U alone: 2.22, 3.65, 9.85, 0.705). The P = 2 figures are
// without the queries' own scales: those are 0.06 ms of a 12.1 ms pass, and 0.12 as a second split of dS instead of a multiplication.
template <int HD, int P, int MAXT, int BLOCKS, bool ONCE>
__global__ void __launch_bounds__(MAXT, BLOCKS) k_attn_bwd_f16(AttnArgs p) {
  after_previous();
  constexpr int KS = HD / 16;
  // The A operands of a block stay in registers over the whole loop where they are few enough; else each step's are loaded
  // where they are used.
  constexpr bool KEEP = HD * P <= 32;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ uint32_t s_max[4], s_vnorm, s_gnorm;  // of Q, K, V, dO
  const int n = blockIdx.x / p.H, h = blockIdx.x % p.H, D = p.H * HD;
  const int e0 = p.off[n], cnt = p.off[n + 1] - e0 + 1;
  const int S16 = round16(cnt), SM = round16(p.S);
  constexpr int PB = pitch<HD, P>();
  const int PV = ONCE ? shared_pitch<HD, P>(SM) : PB;
  uint8_t *sq = smem, *sk = sq + SM * PB, *sg = sk + SM * PB, *sv = sg + SM * PB;
  float *slc = reinterpret_cast<float*>(sv + SM * PV), *sm = slc + SM, *sl = sm + SM, *sd = sl + SM, *sn = sd + SM, *su = sn + SM;  // (su: ONCE)
  // Staging: a thread's loads of U rows' pieces (of all its rows, up to five blocks) are all under way before it looks for the tile's scales or splits any. The
  // HD / 4 lanes that hold a row of dO, V and O add up its Dq = dO . O and its norms on the way.
  constexpr int Q = HD / 4, U = MAXT <= 160 && HD <= 32 ? 4 : 2;
  float4 x0[U], x1[U], x2[U], x3[U], x4[U];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * blockDim.x, r = t / Q;
      const size_t row = r == 0 ? size_t(n) : size_t(p.N) + e0 + r - 1;
      const size_t at = row * 3 * D + h * HD + (t % Q) * 4, ag = row * D + h * HD + (t % Q) * 4;
      x0[u] = get(p.qkv, at, r < cnt), x1[u] = get(p.qkv, at + D, r < cnt), x2[u] = get(p.qkv, at + 2 * D, r < cnt);
      x3[u] = get(p.dmerged, ag, r < cnt), x4[u] = get(p.merged, ag, r < cnt);
    }
  };
  fetch(threadIdx.x);
  if (threadIdx.x < 4) s_max[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_vnorm = s_gnorm = 0;
  for (int r = threadIdx.x; r < S16; r += blockDim.x) {
    float lc = kOff, m = 1e30f, il = 0.f;
    if (r < cnt) {
      const size_t row = r == 0 ? size_t(n) : size_t(p.N) + e0 + r - 1;
      const float cf = r == 0 ? 1.0f : p.cut[e0 + r - 1];
      const float2 ml = *reinterpret_cast<const float2*>(p.ml + (row * p.H + h) * 2);
      lc = cf > 0.f ? __logf(cf) * kLog2e : kOff;
      il = ml.y;
      if (il > 0.f) m = ml.x * kLog2e;  // a dead query's weights are exp(-1e30) = 0
    }
    slc[r] = lc, sm[r] = m, sl[r] = il * 32768.f;
  }
  __syncthreads();
  {
    float mq = 0.f, mk = 0.f, mv = 0.f, mg = 0.f;
    for (int t = threadIdx.x + U * blockDim.x; t < cnt * Q; t += blockDim.x) {
      const int r = t / Q;
      const size_t row = r == 0 ? size_t(n) : size_t(p.N) + e0 + r - 1, at = row * 3 * D + h * HD + (t % Q) * 4;
      mq = max_abs(mq, get(p.qkv, at, true)), mk = max_abs(mk, get(p.qkv, at + D, true)), mv = max_abs(mv, get(p.qkv, at + 2 * D, true));
      mg = max_abs(mg, get(p.dmerged, row * D + h * HD + (t % Q) * 4, true));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) mq = max_abs(mq, x0[u]), mk = max_abs(mk, x1[u]), mv = max_abs(mv, x2[u]), mg = max_abs(mg, x3[u]);
    raise_tile(s_max, mq), raise_tile(s_max + 1, mk), raise_tile(s_max + 2, mv), raise_tile(s_max + 3, mg);
  }
  __syncthreads();
  const float scq = scale_of(s_max[0]), sck = scale_of(s_max[1]), scv = scale_of(s_max[2]), scg = scale_of(s_max[3]);
  const float usq = unscale_of(s_max[0]), usk = unscale_of(s_max[1]), usv = unscale_of(s_max[2]), usg = unscale_of(s_max[3]);
  for (int t0 = threadIdx.x; t0 < S16 * Q; t0 += U * blockDim.x) {
    if (t0 != threadIdx.x) fetch(t0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * blockDim.x, r = t / Q, c = (t % Q) * 4;
      if (t >= S16 * Q) break;  // whole warps: a row block of 16 is 16 Q threads
      const float4 v = x2[u] * scv, go = x3[u] * scg;
      put<HD, P>(sq, r, c, x0[u] * scq), put<HD, P>(sk, r, c, x1[u] * sck), put<HD, P>(sv, r, c, v, PV), put<HD, P>(sg, r, c, go);
      float d = dot4(go, x4[u]), gg = dot4(go, go), vv = dot4(v, v);
#pragma unroll
      for (int o = Q / 2; o > 0; o >>= 1) {
        d += __shfl_xor_sync(0xffffffffu, d, o), gg += __shfl_xor_sync(0xffffffffu, gg, o), vv += __shfl_xor_sync(0xffffffffu, vv, o);
      }
      if (c == 0) {
        sd[r] = d * scv, sn[r] = sqrtf(gg);  // in the units of the scaled products
        atomicMax(&s_vnorm, __float_as_uint(vv)), atomicMax(&s_gnorm, __float_as_uint(gg));
      }
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, g = lane >> 2, t = lane & 3;
  const uint32_t aq = smem_u32(sq), ak = smem_u32(sk), av = smem_u32(sv), ag = smem_u32(sg);
  const float f = usq * usk * p.sc * kLog2e;  // a scaled score product to a score, base 2
  const float vmax = sqrtf(__uint_as_float(s_vnorm)), gmax = sqrtf(__uint_as_float(s_gnorm));
  const int nb = S16 / 16;
  if constexpr (ONCE) {
    {  // a query's own scale (P = 3: over the common one), and the common one over it
      const float all_bound = fmaxf(2.1f * gmax * vmax, 1e-9f);
      // P = 1, 2: at most 2^24 from the common one. The factor that takes a row's parts there for dK is an fp16 number: 2^-25 would be
      // zero and the row missing. dQ keeps its bits down to rows of 2^-40, and dO itself is not staged any finer.
      const float least = P <= 2 ? all_bound * 0x1p-24f : 0.f;
      const uint32_t all = __float_as_uint(all_bound);
      for (int r = threadIdx.x; r < S16; r += blockDim.x) {
        const uint32_t own = __float_as_uint(fmaxf(2.1f * sn[r] * vmax, fmaxf(least, 1e-9f)));
        sn[r] = scale_of(own) * (P == 3 ? unscale_of(all) : 1.f / 32768.f), su[r] = unscale_of(own) * scale_of(all);
      }
      __syncthreads();
    }
    const int r0 = 16 * warp, i0 = r0 + g, i1 = r0 + g + 8;  // this lane's two rows: keys, then queries
    const size_t g0 = i0 == 0 ? size_t(n) : size_t(p.N) + e0 + i0 - 1, g1 = size_t(p.N) + e0 + i1 - 1;
    const uint32_t bound = __float_as_uint(fmaxf(2.1f * gmax * vmax, 1e-9f));  // |dP - D| at most: brings dS to 2^15 (see below)
    if (warp < nb) {
      uint32_t kf[KS][P][4], vf[KS][P][4];
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int j = 0; j < P; ++j) {
          load_a<HD, P>(kf[ks][j], ak, r0, ks, j, lane);
          ldsm4(vf[ks][j], av + (r0 + (lane & 15)) * PV + j * HD * 2 + ks * 32 + (lane >> 4) * 16);
        }
      __syncwarp();
      const float lc0 = slc[i0], lc1 = slc[i1];
      const float ds = scale_of(bound) * (1.f / 32768.f), fds = usv * unscale_of(bound) * usg;
      float dk[HD / 8][4], dv[HD / 8][4];
      clear<HD>(dk), clear<HD>(dv);
      float cf0 = 0.f, cf1 = 0.f;
      for (int b = 0; b < S16; b += 16) {
        Acc<P, 2> c, w;
        two_products<HD, P, true, true>(c, w, kf, vf, ak, av, r0, aq, ag, b, lane);
        float x[2][4], y[2][4];
        __half2 to_common[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int q = b + 8 * i + 2 * t;  // this lane's two queries of the block
          const float2 m = *reinterpret_cast<const float2*>(sm + q), il = *reinterpret_cast<const float2*>(sl + q),
                       d = *reinterpret_cast<const float2*>(sd + q);
          // probabilities by 2^15, score adjoints by ds (P = 1, 2: by the query's own)
          x[i][0] = exp2_fast(fmaf(c.get(i, 0), f, lc0) - m.x) * il.x, x[i][1] = exp2_fast(fmaf(c.get(i, 1), f, lc0) - m.y) * il.y;
          x[i][2] = exp2_fast(fmaf(c.get(i, 2), f, lc1) - m.x) * il.x, x[i][3] = exp2_fast(fmaf(c.get(i, 3), f, lc1) - m.y) * il.y;
          const float2 own = P <= 2 ? *reinterpret_cast<const float2*>(sn + q) : make_float2(ds, ds);
          y[i][0] = x[i][0] * ((w.get(i, 0) - d.x) * own.x), y[i][1] = x[i][1] * ((w.get(i, 1) - d.y) * own.y);
          y[i][2] = x[i][2] * ((w.get(i, 2) - d.x) * own.x), y[i][3] = x[i][3] * ((w.get(i, 3) - d.y) * own.y);
          if (P <= 2) {
            const float2 u = *reinterpret_cast<const float2*>(su + q);
            to_common[i] = __floats2half2_rn(u.x, u.y);
            cf0 += y[i][0] * u.x + y[i][1] * u.y, cf1 += y[i][2] * u.x + y[i][3] * u.y;
          } else {
            cf0 += y[i][0] + y[i][1], cf1 += y[i][2] + y[i][3];
          }
        }
        uint32_t a[with_sum<P>()][4];
        make_a<P>(a, y);
        if (P <= 2) {  // dK sums over the queries, so wants them on one scale: the parts times a power of two, at most 1
          uint32_t k[P][4];
#pragma unroll
          for (int j = 0; j < P; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __half2 v = __hmul2(*reinterpret_cast<const __half2*>(&a[j][i]), to_common[i / 2]);
              k[j][i] = *reinterpret_cast<const uint32_t*>(&v);
            }
          product_rows<HD, P>(dk, k, aq, b, lane);
        } else {
          product_rows<HD, P>(dk, a, aq, b, lane);
        }
        if (P == 3) {  // dQ wants a query's row of dS on the scale of the row's own largest value
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float2 o = *reinterpret_cast<const float2*>(sn + b + 8 * i + 2 * t);
            y[i][0] *= o.x, y[i][1] *= o.y, y[i][2] *= o.x, y[i][3] *= o.y;
          }
          make_a<P>(a, y);
        }
#pragma unroll
        for (int j = 0; j < P; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint8_t* at = sv + size_t(i0) * PV + j * SM * 2 + (b + 8 * i + 2 * t) * 2;
            *reinterpret_cast<uint32_t*>(at) = a[j][2 * i], *reinterpret_cast<uint32_t*>(at + 8 * PV) = a[j][2 * i + 1];
          }
        make_a<P>(a, x);
        product_rows<HD, P>(dv, a, ag, b, lane);
      }
      cf0 += __shfl_xor_sync(0xffffffffu, cf0, 1), cf0 += __shfl_xor_sync(0xffffffffu, cf0, 2);
      cf1 += __shfl_xor_sync(0xffffffffu, cf1, 1), cf1 += __shfl_xor_sync(0xffffffffu, cf1, 2);
      write_rows<HD>(p.qkv_adj, 3 * D, D + h * HD, g0, g1, i0 < cnt, i1 < cnt, dk, fds * usq * p.sc, fds * usq * p.sc, p.qkv_adj_max, t);
      write_rows<HD>(p.qkv_adj, 3 * D, 2 * D + h * HD, g0, g1, i0 < cnt, i1 < cnt, dv, usg * (1.f / 32768.f), usg * (1.f / 32768.f),
                     p.qkv_adj_max, t);
      if (t == 0) {  // each key's dS summed over its queries: the cutoff factor's share from this head
        if (i0 < cnt) p.cfh[g0 * p.H + h] = cf0 * fds;
        if (i1 < cnt) p.cfh[g1 * p.H + h] = cf1 * fds;
      }
    }
    __syncthreads();
    if (warp >= nb) return;
    float dq[HD / 8][4];
    clear<HD>(dq);
    for (int b = 0; b < S16; b += 16) {
      uint32_t a[with_sum<P>()][4];
#pragma unroll
      for (int j = 0; j < P; ++j)  // 8 x 8 blocks of dS^T, keys down, turned: rows of 16 queries, 16 keys of the contraction
        ldsm4_t(a[j], av + (b + (lane >> 4) * 8 + (lane & 7)) * PV + j * SM * 2 + (r0 + ((lane >> 3) & 1) * 8) * 2);
      add_sum<P>(a);
      product_rows<HD, P>(dq, a, ak, b, lane);
    }
    const float fdq = usv * usk * usg * p.sc * unscale_of(bound), f0 = fdq * su[i0], f1 = fdq * su[i1];
    write_rows<HD>(p.qkv_adj, 3 * D, h * HD, g0, g1, i0 < cnt, i1 < cnt, dq, f0, f1, p.qkv_adj_max, t);
    return;
  }
  for (int task = warp; task < 2 * nb; task += nw) {
    const bool keys = task >= nb;
    const int r0 = 16 * (keys ? task - nb : task);
    const int i0 = r0 + g, i1 = r0 + g + 8;  // this lane's two rows (queries or keys)
    const size_t g0 = i0 == 0 ? size_t(n) : size_t(p.N) + e0 + i0 - 1, g1 = size_t(p.N) + e0 + i1 - 1;
    uint32_t a1[KEEP ? KS : 1][P][4], a2[KEEP ? KS : 1][P][4];
    if (KEEP) {
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int j = 0; j < P; ++j) {
          load_a<HD, P>(a1[KEEP ? ks : 0][j], keys ? ak : aq, r0, ks, j, lane);
          load_a<HD, P>(a2[KEEP ? ks : 0][j], keys ? av : ag, r0, ks, j, lane);
        }
    }
    if (!keys) {
      // |dP - D| of a query is at most twice its |dO| times the largest |V|: that brings its row of dS to 2^15. Not below
      // 1e-9, or a norm whose squares have vanished would let what is left of its row past fp16's range.
      const uint32_t b0 = __float_as_uint(fmaxf(2.1f * sn[i0] * vmax, 1e-9f)), b1 = __float_as_uint(fmaxf(2.1f * sn[i1] * vmax, 1e-9f));
      const float m0 = sm[i0], m1 = sm[i1], il0 = sl[i0] * (1.f / 32768.f) * scale_of(b0), il1 = sl[i1] * (1.f / 32768.f) * scale_of(b1), d0 = sd[i0], d1 = sd[i1];
      float dq[HD / 8][4];
      clear<HD>(dq);
      for (int b = 0; b < S16; b += 16) {
        if (!KEEP) asm volatile("" ::: "memory");  // or the loads of the A operands are hoisted and live across the loop again
        Acc<P, 2> c, w;
        two_products<HD, P, KEEP, true>(c, w, a1, a2, aq, ag, r0, ak, av, b, lane);
        float x[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 lc = *reinterpret_cast<const float2*>(slc + b + 8 * i + 2 * t);
          x[i][0] = exp2_fast(fmaf(c.get(i, 0), f, lc.x) - m0) * il0 * (w.get(i, 0) - d0);
          x[i][1] = exp2_fast(fmaf(c.get(i, 1), f, lc.y) - m0) * il0 * (w.get(i, 1) - d0);
          x[i][2] = exp2_fast(fmaf(c.get(i, 2), f, lc.x) - m1) * il1 * (w.get(i, 2) - d1);
          x[i][3] = exp2_fast(fmaf(c.get(i, 3), f, lc.y) - m1) * il1 * (w.get(i, 3) - d1);
        }
        uint32_t a[with_sum<P>()][4];
        make_a<P>(a, x);
        product_rows<HD, P>(dq, a, ak, b, lane);
      }
      write_rows<HD>(p.qkv_adj, 3 * D, h * HD, g0, g1, i0 < cnt, i1 < cnt, dq, usv * usk * p.sc * unscale_of(b0) * usg, usv * usk * p.sc * unscale_of(b1) * usg,
                        p.qkv_adj_max, t);
    } else {
      // transposed: rows are keys. S^T = K Q^T and dP^T = V dO^T per block of 16 queries
      const float lc0 = slc[i0], lc1 = slc[i1];
      const uint32_t bound = __float_as_uint(fmaxf(2.1f * gmax * vmax, 1e-9f));
      const float ds = scale_of(bound) * (1.f / 32768.f), fds = usv * unscale_of(bound) * usg;
      float dk[HD / 8][4], dv[HD / 8][4];
      clear<HD>(dk), clear<HD>(dv);
      float cf0 = 0.f, cf1 = 0.f;
      for (int b = 0; b < S16; b += 16) {
        if (!KEEP) asm volatile("" ::: "memory");
        Acc<P, 2> c, w;
        two_products<HD, P, KEEP, true>(c, w, a1, a2, ak, av, r0, aq, ag, b, lane);
        float x[2][4], y[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int q = b + 8 * i + 2 * t;  // this lane's two queries of the block
          const float2 m = *reinterpret_cast<const float2*>(sm + q), il = *reinterpret_cast<const float2*>(sl + q),
                       d = *reinterpret_cast<const float2*>(sd + q);
          // probabilities by 2^15, score adjoints by ds
          x[i][0] = exp2_fast(fmaf(c.get(i, 0), f, lc0) - m.x) * il.x, x[i][1] = exp2_fast(fmaf(c.get(i, 1), f, lc0) - m.y) * il.y;
          x[i][2] = exp2_fast(fmaf(c.get(i, 2), f, lc1) - m.x) * il.x, x[i][3] = exp2_fast(fmaf(c.get(i, 3), f, lc1) - m.y) * il.y;
          y[i][0] = x[i][0] * ((w.get(i, 0) - d.x) * ds), y[i][1] = x[i][1] * ((w.get(i, 1) - d.y) * ds);
          y[i][2] = x[i][2] * ((w.get(i, 2) - d.x) * ds), y[i][3] = x[i][3] * ((w.get(i, 3) - d.y) * ds);
          cf0 += y[i][0] + y[i][1], cf1 += y[i][2] + y[i][3];
        }
        uint32_t a[with_sum<P>()][4];
        make_a<P>(a, y);
        product_rows<HD, P>(dk, a, aq, b, lane);
        make_a<P>(a, x);
        product_rows<HD, P>(dv, a, ag, b, lane);
      }
      cf0 += __shfl_xor_sync(0xffffffffu, cf0, 1), cf0 += __shfl_xor_sync(0xffffffffu, cf0, 2);
      cf1 += __shfl_xor_sync(0xffffffffu, cf1, 1), cf1 += __shfl_xor_sync(0xffffffffu, cf1, 2);
      write_rows<HD>(p.qkv_adj, 3 * D, D + h * HD, g0, g1, i0 < cnt, i1 < cnt, dk, fds * usq * p.sc, fds * usq * p.sc, p.qkv_adj_max, t);
      write_rows<HD>(p.qkv_adj, 3 * D, 2 * D + h * HD, g0, g1, i0 < cnt, i1 < cnt, dv, usg * (1.f / 32768.f), usg * (1.f / 32768.f),
                        p.qkv_adj_max, t);
      if (t == 0) {  // each key's dS summed over its queries: the cutoff factor's share from this head
        if (i0 < cnt) p.cfh[g0 * p.H + h] = cf0 * fds;
        if (i1 < cnt) p.cfh[g1 * p.H + h] = cf1 * fds;
      }
    }
  }
}

template <class K>
void launch(Stream& st, K kernel, const AttnArgs& p, size_t bytes, int threads, SmemOptIn& opted) {
  opt_in_shared_memory(kernel, bytes, opted);
  launch(st, kernel, p.N * p.H, threads, bytes, p);
  PETB_LAUNCH_CHECK(st);
}

constexpr size_t kMaxBytes = 224 * 1024;

template <int HD, int P>
bool fwd_hd(Stream& st, const AttnArgs& p) {
  const int blocks = round16(p.S) / 16;
  const size_t bytes = size_t(round16(p.S)) * (3 * pitch<HD, P>() + sizeof(float));
  if (blocks > 11 || bytes > kMaxBytes) return false;
  static SmemOptIn o2, o5, o8, o11;
  if (blocks <= 2) launch(st, k_attn_fwd_f16<HD, P, 2>, p, bytes, 32 * blocks, o2);
  else if (blocks <= 5) launch(st, k_attn_fwd_f16<HD, P, 5>, p, bytes, 32 * blocks, o5);
  else if (blocks <= 8) launch(st, k_attn_fwd_f16<HD, P, 8>, p, bytes, 32 * blocks, o8);
  else launch(st, k_attn_fwd_f16<HD, P, 11>, p, bytes, 32 * blocks, o11);
  return true;
}
template <int HD, int P>
bool bwd_hd(Stream& st, const AttnArgs& p) {
  const int rows = round16(p.S), blocks = rows / 16;
  const size_t bytes = size_t(rows) * (4 * pitch<HD, P>() + 5 * sizeof(float));
  if (bytes > kMaxBytes) return false;
  static SmemOptIn o128, o160, o320, o640;
  // Up to five blocks of 16 rows, heads of at most 32: scores once (a head size of 64 has no registers for two tensors' operands).
  if constexpr (HD <= 32) {
    if (blocks <= 5) {
      const size_t once = size_t(rows) * (3 * pitch<HD, P>() + shared_pitch<HD, P>(rows) + 6 * sizeof(float));
      if (blocks <= 4) launch(st, k_attn_bwd_f16<HD, P, 128, P == 3 ? 3 : P == 2 ? 4 : 5, true>, p, once, 32 * blocks, o128);
      else launch(st, k_attn_bwd_f16<HD, P, 160, P == 3 ? 2 : P == 2 ? 3 : 4, true>, p, once, 32 * blocks, o160);
      return true;
    }
  } else if (blocks <= 5) {
    launch(st, k_attn_bwd_f16<HD, P, 160, resident<HD, P, 4>(80), false>, p, bytes, 32 * blocks, o160);
    return true;
  }
  // A warp per 16 rows, which takes queries and then keys, where several CTAs share an SM; where one tile fills it, a warp
  // per 16 queries and one per 16 keys, up to 20: then blocks in turn.
  if (bytes <= 110 * 1024) launch(st, k_attn_bwd_f16<HD, P, 320, 2, false>, p, bytes, 32 * (blocks < 10 ? blocks : 10), o320);
  else launch(st, k_attn_bwd_f16<HD, P, 640, 1, false>, p, bytes, 64 * (blocks < 10 ? blocks : 10), o640);
  return true;
}
template <int P>
bool fwd_p(Stream& st, const AttnArgs& p) {
  switch (p.hd) {
    case 16: return fwd_hd<16, P>(st, p);
    case 32: return fwd_hd<32, P>(st, p);
    case 64: return fwd_hd<64, P>(st, p);
    default: return false;
  }
}
template <int P>
bool bwd_p(Stream& st, const AttnArgs& p) {
  switch (p.hd) {
    case 16: return bwd_hd<16, P>(st, p);
    case 32: return bwd_hd<32, P>(st, p);
    case 64: return bwd_hd<64, P>(st, p);
    default: return false;
  }
}

}  // namespace

// True if these kernels took the pass; false leaves it to the others (an atom with too many tokens, another head size).
bool attention_forward_f16(Stream& st, const AttnArgs& p) {
  return p.mode == ATTN_NATIVE ? fwd_p<3>(st, p) : p.mode == ATTN_TF32X3 ? fwd_p<2>(st, p) : fwd_p<1>(st, p);
}
bool attention_backward_f16(Stream& st, const AttnArgs& p) {
  return p.mode == ATTN_NATIVE ? bwd_p<3>(st, p) : p.mode == ATTN_TF32X3 ? bwd_p<2>(st, p) : bwd_p<1>(st, p);
}

}  // namespace petb
