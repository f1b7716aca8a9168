// The network's non-GEMM passes: see ops.h.
#include "ops.h"

#include "epilogue.cuh"

namespace petb {

namespace {

constexpr float kLnEps = 1e-5f;                     // kLayerNormEps (:196)
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ float max4(const float4& v) { return max_abs4(v.x, v.y, v.z, v.w); }

// Row r's largest magnitude raised to m, for kernels with a thread per run of four of a row's D4 runs: where a row is whole
// warps, a warp's largest goes out once.
__device__ __forceinline__ void raise_row(uint32_t* mx, int r, int D4, float m) {
  if (!mx) return;
  if (D4 % 32 == 0) {
    m = warp_max(m);
    if (threadIdx.x % 32) return;
  }
  atomicMax(mx + r, __float_as_uint(m));
}

// out(r, :) = table(idx(r), :). Two tables' lookups in one launch: blocks from `blocks0` on do the second's.
struct Lookup {
  float* out;
  const float* table;
  const int* idx;
  uint32_t* mx;
  int R, D4;
};
__global__ void k_gather_rows(Lookup first, Lookup second, int blocks0) {
  after_previous();
  const bool one = int(blockIdx.x) < blocks0;
  const Lookup& p = one ? first : second;
  const size_t t = size_t(blockIdx.x - (one ? 0 : blocks0)) * blockDim.x + threadIdx.x;
  if (t >= size_t(p.R) * p.D4) return;
  const int r = int(t / p.D4), q = int(t % p.D4);
  const float4 v = reinterpret_cast<const float4*>(p.table)[size_t(p.idx[r]) * p.D4 + q];
  reinterpret_cast<float4*>(p.out)[t] = v;
  raise_row(p.mx, r, p.D4, max4(v));
}

// A thread has four columns of `rows` neighbouring rows: the columns' weights (64 bytes a column, four times what it writes of a
// row) are read once for all of them. 120314 x 256: 104 us with a row a thread, 56 with eight; 38 at HBM's rate.
__global__ void __launch_bounds__(256) k_compress0(GemmArgs p, int rows) {
  after_previous();
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int D4 = p.N / 4, col = int(t % D4) * 4;
  const size_t first = t / D4 * rows;
  if (first >= size_t(p.M)) return;
  const float4 b = ld4(p.bias + col);
  float4 w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = ld4(p.wx + size_t(col + j) * 4);
  const size_t end = first + rows < size_t(p.M) ? first + rows : size_t(p.M);
#pragma unroll 2
  for (size_t row = first; row < end; ++row) {
    const float4 tt = ld4(p.tab + size_t(p.sp[row]) * p.N + col);
    const float e0 = (float) p.vec[3 * row], e1 = (float) p.vec[3 * row + 1], e2 = (float) p.vec[3 * row + 2], e3 = (float) p.dist[row];
    float z[4] = {b.x, b.y, b.z, b.w};
    const float from_table[4] = {tt.x, tt.y, tt.z, tt.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) z[j] = z[j] + from_table[j] + w[j].x * e0 + w[j].y * e1 + w[j].z * e2 + w[j].w * e3;
    st4(p.pre + row * p.ldp + col, make_float4(z[0], z[1], z[2], z[3]));
    const float4 o = make_float4(silu_f(z[0]), silu_f(z[1]), silu_f(z[2]), silu_f(z[3]));
    st4(p.C + row * p.ldc + col, o);
    raise_row(p.c_max, int(row), D4, max_abs4(o.x, o.y, o.z, o.w));
  }
}

// One warp per row. x = in (+ add, stored back); out = (x - mu) inv w + b.
__global__ void __launch_bounds__(256) k_norm_fwd(float* __restrict__ out, float* __restrict__ in, const float* __restrict__ add,
                                                  const float* __restrict__ w, const float* __restrict__ bias, int R, int D,
                                                  uint32_t* __restrict__ mx) {
  after_previous();
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= R) return;
  float* x = in + size_t(r) * D;
  const bool ln = bias != nullptr;
  if (add) {
    const float* a = add + size_t(r) * D;
    for (int d = lane; d < D; d += 32) x[d] += a[d];
  }
  float mu = 0.f;
  if (ln) {
    float s = 0.f;
    for (int d = lane; d < D; d += 32) s += x[d];
    mu = warp_sum(s) / D;
  }
  float v = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float c = x[d] - mu;
    v += c * c;
  }
  v = warp_sum(v);
  const float inv = 1.0f / sqrtf(v / D + (ln ? kLnEps : kRmsEps));
  float* o = out + size_t(r) * D;
  float big = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float y = (x[d] - mu) * inv * w[d] + (ln ? bias[d] : 0.f);
    o[d] = y, big = fmaxf(big, fabsf(y));
  }
  if (!mx) return;
  big = warp_max(big);
  if (lane == 0) mx[r] = __float_as_uint(big);
}

// Edge q's partner row: its reverse edge's, the row another rank sent for it, or none.
__device__ __forceinline__ const float* partner_row(const float* oe, const int* rev, const RemoteRows& rm, int q, int D) {
  const int r = rev[q];
  if (r >= 0) return oe + size_t(r) * D;
  if (rm.of) {
    const int l = rm.of[q];
    if (l >= 0) return rm.rows + size_t(l) * D;
  }
  return nullptr;
}

__global__ void k_gather_live(float* __restrict__ out, const float* __restrict__ src, int ld, int col0,
                              const int* __restrict__ live_packed, int n_live, int D4) {
  after_previous();
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= size_t(n_live) * D4) return;
  const int l = int(t / D4), q = int(t % D4), k = live_packed[l];
  reinterpret_cast<float4*>(out)[t] = k >= 0 ? ld4(src + size_t(k) * ld + col0 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// The same with each lane holding NV runs of four consecutive values in registers (D = 128 NV): the row is read
// once, 16 bytes at a time, for the statistics and for the output.
template <int NV>
__global__ void __launch_bounds__(256) k_norm_fwd_v(float* __restrict__ out, float* __restrict__ in, const float* __restrict__ add,
                                                    const float* __restrict__ w, const float* __restrict__ bias, int R,
                                                    uint32_t* __restrict__ mx) {
  after_previous();
  constexpr int D = 128 * NV;
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= R) return;
  float* x = in + size_t(r) * D;
  const bool ln = bias != nullptr;
  float4 v[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = ld4(x + 128 * i + 4 * lane);
  if (add) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const float4 a = ld4(add + size_t(r) * D + 128 * i + 4 * lane);
      v[i].x += a.x, v[i].y += a.y, v[i].z += a.z, v[i].w += a.w;
      st4(x + 128 * i + 4 * lane, v[i]);
    }
  }
  float mu = 0.f;
  if (ln) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    mu = warp_sum(s) / D;
  }
  float q = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const float a = v[i].x - mu, b = v[i].y - mu, c = v[i].z - mu, d = v[i].w - mu;
    q += (a * a + b * b) + (c * c + d * d);
  }
  q = warp_sum(q);
  const float inv = 1.0f / sqrtf(q / D + (ln ? kLnEps : kRmsEps));
  float* o = out + size_t(r) * D;
  float big = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const float4 ww = ld4(w + 128 * i + 4 * lane);
    float4 y = make_float4((v[i].x - mu) * inv * ww.x, (v[i].y - mu) * inv * ww.y, (v[i].z - mu) * inv * ww.z,
                           (v[i].w - mu) * inv * ww.w);
    if (ln) {
      const float4 bb = ld4(bias + 128 * i + 4 * lane);
      y.x += bb.x, y.y += bb.y, y.z += bb.z, y.w += bb.w;
    }
    st4(o + 128 * i + 4 * lane, y);
    big = fmaxf(big, max4(y));
  }
  if (!mx) return;
  big = warp_max(big);
  if (lane == 0) mx[r] = __float_as_uint(big);
}

__global__ void __launch_bounds__(256) k_concat_norm_fwd(float* __restrict__ out, const float* __restrict__ oe,
                                                         const int* __restrict__ rev, float* __restrict__ ie,
                                                         const float* __restrict__ w, const float* __restrict__ bias, int E,
                                                         int D, RemoteRows rm, uint32_t* __restrict__ mx) {
  after_previous();
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (k >= E) return;
  const int W = 2 * D;
  const float* a = oe + size_t(k) * D;
  const float* b = partner_row(oe, rev, rm, k, D);
  float s = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float v = a[d];
    ie[size_t(k) * D + d] += v;
    s += v + (b ? b[d] : 0.f);
  }
  const float mu = warp_sum(s) / W;
  float v = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float c0 = a[d] - mu, c1 = (b ? b[d] : 0.f) - mu;
    v += c0 * c0 + c1 * c1;
  }
  v = warp_sum(v);
  const float inv = 1.0f / sqrtf(v / W + kLnEps);
  float* o = out + size_t(k) * W;
  float big = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float y0 = (a[d] - mu) * inv * w[d] + bias[d], y1 = ((b ? b[d] : 0.f) - mu) * inv * w[D + d] + bias[D + d];
    o[d] = y0, o[D + d] = y1;
    big = fmaxf(big, fmaxf(fabsf(y0), fabsf(y1)));
  }
  if (!mx) return;
  big = warp_max(big);
  if (lane == 0) mx[k] = __float_as_uint(big);
}

struct RowStats {
  float mu, inv, mg, mgx;
};

__global__ void __launch_bounds__(256) k_norm_bwd(float* __restrict__ in_adj, const float* __restrict__ out_adj,
                                                  const float* __restrict__ in, const float* __restrict__ w, bool ln, int R, int D,
                                                  int acc_row0, float* __restrict__ also, uint32_t* __restrict__ mx) {
  after_previous();
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= R) return;
  const float* x = in + size_t(r) * D;
  const float* ga = out_adj + size_t(r) * D;
  float mu = 0.f;
  if (ln) {
    float s = 0.f;
    for (int d = lane; d < D; d += 32) s += x[d];
    mu = warp_sum(s) / D;
  }
  float sq = 0.f, sg = 0.f, sgx = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float c = x[d] - mu, gw = w ? ga[d] * w[d] : ga[d];
    sq += c * c, sg += gw, sgx += gw * c;
  }
  sq = warp_sum(sq), sg = warp_sum(sg), sgx = warp_sum(sgx);
  const float inv = 1.0f / sqrtf(sq / D + (ln ? kLnEps : kRmsEps));
  const float mg = ln ? sg / D : 0.f, mgx = sgx * inv / D;
  float* o = in_adj + size_t(r) * D;
  const bool acc = r >= acc_row0;
  float big = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float g = inv * ((w ? ga[d] * w[d] : ga[d]) - mg - (x[d] - mu) * inv * mgx);
    const float v = acc ? o[d] + g : g;
    o[d] = v;
    if (also) also[size_t(r) * D + d] = v;
    big = fmaxf(big, fabsf(v));
  }
  if (!mx) return;
  big = warp_max(big);
  if (lane == 0) mx[r] = __float_as_uint(big);
}

template <int NV>
__global__ void __launch_bounds__(256) k_norm_bwd_v(float* __restrict__ in_adj, const float* __restrict__ out_adj,
                                                    const float* __restrict__ in, const float* __restrict__ w, bool ln, int R,
                                                    int acc_row0, float* __restrict__ also, uint32_t* __restrict__ mx) {
  after_previous();
  constexpr int D = 128 * NV;
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= R) return;
  float4 x[NV], gw[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    x[i] = ld4(in + size_t(r) * D + 128 * i + 4 * lane);
    gw[i] = ld4(out_adj + size_t(r) * D + 128 * i + 4 * lane);
    if (w) {
      const float4 ww = ld4(w + 128 * i + 4 * lane);
      gw[i].x *= ww.x, gw[i].y *= ww.y, gw[i].z *= ww.z, gw[i].w *= ww.w;
    }
  }
  float mu = 0.f;
  if (ln) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) s += (x[i].x + x[i].y) + (x[i].z + x[i].w);
    mu = warp_sum(s) / D;
  }
  float sq = 0.f, sg = 0.f, sgx = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    x[i].x -= mu, x[i].y -= mu, x[i].z -= mu, x[i].w -= mu;
    sq += (x[i].x * x[i].x + x[i].y * x[i].y) + (x[i].z * x[i].z + x[i].w * x[i].w);
    sg += (gw[i].x + gw[i].y) + (gw[i].z + gw[i].w);
    sgx += (gw[i].x * x[i].x + gw[i].y * x[i].y) + (gw[i].z * x[i].z + gw[i].w * x[i].w);
  }
  sq = warp_sum(sq), sg = warp_sum(sg), sgx = warp_sum(sgx);
  const float inv = 1.0f / sqrtf(sq / D + (ln ? kLnEps : kRmsEps));
  const float mg = ln ? sg / D : 0.f, mgx = sgx * inv / D;
  float* o = in_adj + size_t(r) * D;
  const bool acc = r >= acc_row0;
  float big = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float4 g = make_float4(inv * (gw[i].x - mg - x[i].x * inv * mgx), inv * (gw[i].y - mg - x[i].y * inv * mgx),
                           inv * (gw[i].z - mg - x[i].z * inv * mgx), inv * (gw[i].w - mg - x[i].w * inv * mgx));
    if (acc) {
      const float4 old = ld4(o + 128 * i + 4 * lane);
      g.x += old.x, g.y += old.y, g.z += old.z, g.w += old.w;
    }
    st4(o + 128 * i + 4 * lane, g);
    if (also) st4(also + size_t(r) * D + 128 * i + 4 * lane, g);
    big = fmaxf(big, max4(g));
  }
  if (!mx) return;
  big = warp_max(big);
  if (lane == 0) mx[r] = __float_as_uint(big);
}

// RMSNorm's backward (`w` null for a gain of one) onto the atoms' rows, a block a row, and the edges', a warp a row, in one
// launch: the few atoms' rows by themselves take 5-10 us, as a warp's rows of 1024 columns and more registers they would take the
// edges' loads their warps.
struct NormBwdRows {
  float* in_adj;         // += the adjoint
  const float* out_adj;
  const float* in;
  const float* w;
  uint32_t* mx;
  int R, D;
};
__device__ __forceinline__ float4 with_gain(float4 g, const float* w, int c) {
  if (!w) return g;
  const float4 x = ld4(w + c);
  return make_float4(g.x * x.x, g.y * x.y, g.z * x.z, g.w * x.w);
}
template <int NV>
__global__ void __launch_bounds__(256) k_norm_bwd_two(NormBwdRows n, NormBwdRows e) {
  after_previous();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (int(blockIdx.x) < n.R) {
    __shared__ float s_sq[8], s_gx[8], s_big[8];
    const size_t at = size_t(blockIdx.x) * n.D;
    float4 x[2], g[2];
    float sq = 0.f, sgx = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = 1024 * i + 4 * threadIdx.x;
      x[i] = c < n.D ? ld4(n.in + at + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      g[i] = c < n.D ? with_gain(ld4(n.out_adj + at + c), n.w, c) : make_float4(0.f, 0.f, 0.f, 0.f);
      sq += (x[i].x * x[i].x + x[i].y * x[i].y) + (x[i].z * x[i].z + x[i].w * x[i].w);
      sgx += (g[i].x * x[i].x + g[i].y * x[i].y) + (g[i].z * x[i].z + g[i].w * x[i].w);
    }
    sq = warp_sum(sq), sgx = warp_sum(sgx);
    if (lane == 0) s_sq[warp] = sq, s_gx[warp] = sgx;
    __syncthreads();
    sq = sgx = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) sq += s_sq[w], sgx += s_gx[w];
    const float inv = 1.0f / sqrtf(sq / n.D + kRmsEps), mgx = sgx * inv / n.D;
    float big = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = 1024 * i + 4 * threadIdx.x;
      if (c >= n.D) continue;
      float4 o = ld4(n.in_adj + at + c);
      o.x += inv * (g[i].x - x[i].x * inv * mgx), o.y += inv * (g[i].y - x[i].y * inv * mgx);
      o.z += inv * (g[i].z - x[i].z * inv * mgx), o.w += inv * (g[i].w - x[i].w * inv * mgx);
      st4(n.in_adj + at + c, o);
      big = fmaxf(big, max4(o));
    }
    if (!n.mx) return;
    big = warp_max(big);
    if (lane == 0) s_big[warp] = big;
    __syncthreads();
    if (threadIdx.x) return;
    for (int w = 1; w < 8; ++w) big = fmaxf(big, s_big[w]);
    n.mx[blockIdx.x] = __float_as_uint(big);
    return;
  }
  constexpr int D = 128 * NV;
  const int r = (blockIdx.x - n.R) * 8 + warp;
  if (r >= e.R) return;
  float4 x[NV], g[NV];
  float sq = 0.f, sgx = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = 128 * i + 4 * lane;
    x[i] = ld4(e.in + size_t(r) * D + c), g[i] = with_gain(ld4(e.out_adj + size_t(r) * D + c), e.w, c);
    sq += (x[i].x * x[i].x + x[i].y * x[i].y) + (x[i].z * x[i].z + x[i].w * x[i].w);
    sgx += (g[i].x * x[i].x + g[i].y * x[i].y) + (g[i].z * x[i].z + g[i].w * x[i].w);
  }
  sq = warp_sum(sq), sgx = warp_sum(sgx);
  const float inv = 1.0f / sqrtf(sq / D + kRmsEps), mgx = sgx * inv / D;
  float* o = e.in_adj + size_t(r) * D;
  float big = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float4 old = ld4(o + 128 * i + 4 * lane);
    old.x += inv * (g[i].x - x[i].x * inv * mgx), old.y += inv * (g[i].y - x[i].y * inv * mgx);
    old.z += inv * (g[i].z - x[i].z * inv * mgx), old.w += inv * (g[i].w - x[i].w * inv * mgx);
    st4(o + 128 * i + 4 * lane, old);
    big = fmaxf(big, max4(old));
  }
  if (!e.mx) return;
  big = warp_max(big);
  if (lane == 0) e.mx[r] = __float_as_uint(big);
}

// The statistics of row q of the concat [oe(q) | partner(q) or 0] and of its adjoint.
__device__ __forceinline__ RowStats concat_stats(const float* oe, const float* b, const float* out_adj, const float* w, int q,
                                                 int D, int lane) {
  const int W = 2 * D;
  const float* a = oe + size_t(q) * D;
  const float* ga = out_adj + size_t(q) * W;
  float s = 0.f;
  for (int d = lane; d < D; d += 32) s += a[d] + (b ? b[d] : 0.f);
  const float mu = warp_sum(s) / W;
  float sq = 0.f, sg = 0.f, sgx = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float c0 = a[d] - mu, c1 = (b ? b[d] : 0.f) - mu;
    const float g0 = ga[d] * w[d], g1 = ga[D + d] * w[D + d];
    sq += c0 * c0 + c1 * c1, sg += g0 + g1, sgx += g0 * c0 + g1 * c1;
  }
  sq = warp_sum(sq), sg = warp_sum(sg), sgx = warp_sum(sgx);
  const float inv = 1.0f / sqrtf(sq / W + kLnEps);
  return RowStats{mu, inv, sg / W, sgx * inv / W};
}

__global__ void __launch_bounds__(256) k_concat_norm_bwd(float* __restrict__ edge_adj, const float* __restrict__ out_adj,
                                                         const float* __restrict__ oe, const int* __restrict__ rev,
                                                         const float* __restrict__ ie_adj, const float* __restrict__ w, int E,
                                                         int D, RemoteRows rm, const float* __restrict__ remote_adj,
                                                         uint32_t* __restrict__ mx) {
  after_previous();
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (k >= E) return;
  const int W = 2 * D, r = rev[k];
  const RowStats sk = concat_stats(oe, partner_row(oe, rev, rm, k, D), out_adj, w, k, D, lane);
  RowStats sr = sk;
  const float* xr2 = nullptr;  // the second half of row r: its partner's row
  if (r >= 0) {
    xr2 = partner_row(oe, rev, rm, r, D);
    sr = concat_stats(oe, xr2, out_adj, w, r, D, lane);
  }
  // An edge to another rank's atom: that rank computed the adjoint of the row it read from here.
  const float* far = (r < 0 && rm.of && remote_adj && rm.of[k] >= 0) ? remote_adj + size_t(rm.of[k]) * D : nullptr;
  float big = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float gk = sk.inv * (out_adj[size_t(k) * W + d] * w[d] - sk.mg - (oe[size_t(k) * D + d] - sk.mu) * sk.inv * sk.mgx);
    float back = 0.f;
    if (r >= 0) {
      const float x = (xr2 ? xr2[d] : 0.f) - sr.mu;
      back = sr.inv * (out_adj[size_t(r) * W + D + d] * w[D + d] - sr.mg - x * sr.inv * sr.mgx);
    } else if (far) {
      back = far[d];
    }
    const float v = ie_adj[size_t(k) * D + d] + gk + back;
    edge_adj[size_t(k) * D + d] = v;
    big = fmaxf(big, fabsf(v));
  }
  if (!mx) return;
  big = warp_max(big);
  if (lane == 0) mx[k] = __float_as_uint(big);
}

// The same, one warp per PAIR of partner rows (single-rank lists only). Row k's concat is [oe(k) | oe(r)] and row r's is
// [oe(r) | oe(k)]: the same numbers, so one mean and one variance serve both, and each row is read once for the two
// outputs. The warp of the larger index of a pair leaves; a row without a partner is a pair with a zero half.
template <int NV>
__global__ void __launch_bounds__(256) k_concat_norm_bwd_pair(float* __restrict__ edge_adj, const float* __restrict__ out_adj,
                                                              const float* __restrict__ oe, const int* __restrict__ rev,
                                                              const float* __restrict__ ie_adj, const float* __restrict__ w,
                                                              int E, uint32_t* __restrict__ mx) {
  after_previous();
  constexpr int D = 128 * NV, W = 2 * D;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (k >= E) return;
  const int r = rev[k];
  const bool mutual = r >= 0 && rev[r] == k;
  if (mutual && r < k) return;
  if (r >= 0 && !mutual) {
    // A list whose partner map is not an involution: this row alone, partner's statistics from its own partner.
    const RemoteRows none{};
    const RowStats sk = concat_stats(oe, oe + size_t(r) * D, out_adj, w, k, D, lane);
    const float* xr2 = partner_row(oe, rev, none, r, D);
    const RowStats sr = concat_stats(oe, xr2, out_adj, w, r, D, lane);
    float big = 0.f;
    for (int d = lane; d < D; d += 32) {
      const float gk = sk.inv * (out_adj[size_t(k) * W + d] * w[d] - sk.mg - (oe[size_t(k) * D + d] - sk.mu) * sk.inv * sk.mgx);
      const float x = (xr2 ? xr2[d] : 0.f) - sr.mu;
      const float back = sr.inv * (out_adj[size_t(r) * W + D + d] * w[D + d] - sr.mg - x * sr.inv * sr.mgx);
      const float v = ie_adj[size_t(k) * D + d] + gk + back;
      edge_adj[size_t(k) * D + d] = v;
      big = fmaxf(big, fabsf(v));
    }
    if (mx) {
      big = warp_max(big);
      if (lane == 0) mx[k] = __float_as_uint(big);
    }
    return;
  }
  float4 a[NV], b[NV], g0[NV], g1[NV], h0[NV], h1[NV];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = 128 * i + 4 * lane;
    a[i] = ld4(oe + size_t(k) * D + c);
    b[i] = mutual ? ld4(oe + size_t(r) * D + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 w0 = ld4(w + c), w1 = ld4(w + D + c);
    const float4 p = ld4(out_adj + size_t(k) * W + c), q = ld4(out_adj + size_t(k) * W + D + c);
    g0[i] = make_float4(p.x * w0.x, p.y * w0.y, p.z * w0.z, p.w * w0.w);
    g1[i] = make_float4(q.x * w1.x, q.y * w1.y, q.z * w1.z, q.w * w1.w);
    if (mutual) {
      const float4 t = ld4(out_adj + size_t(r) * W + c), u = ld4(out_adj + size_t(r) * W + D + c);
      h0[i] = make_float4(t.x * w0.x, t.y * w0.y, t.z * w0.z, t.w * w0.w);
      h1[i] = make_float4(u.x * w1.x, u.y * w1.y, u.z * w1.z, u.w * w1.w);
    } else {
      h0[i] = h1[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    s += ((a[i].x + b[i].x) + (a[i].y + b[i].y)) + ((a[i].z + b[i].z) + (a[i].w + b[i].w));
  }
  const float mu = warp_sum(s) / W;
  float sq = 0.f, sgk = 0.f, sgxk = 0.f, sgr = 0.f, sgxr = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    a[i].x -= mu, a[i].y -= mu, a[i].z -= mu, a[i].w -= mu;
    b[i].x -= mu, b[i].y -= mu, b[i].z -= mu, b[i].w -= mu;
    sq += ((a[i].x * a[i].x + b[i].x * b[i].x) + (a[i].y * a[i].y + b[i].y * b[i].y)) +
          ((a[i].z * a[i].z + b[i].z * b[i].z) + (a[i].w * a[i].w + b[i].w * b[i].w));
    sgk += ((g0[i].x + g1[i].x) + (g0[i].y + g1[i].y)) + ((g0[i].z + g1[i].z) + (g0[i].w + g1[i].w));
    sgxk += ((g0[i].x * a[i].x + g1[i].x * b[i].x) + (g0[i].y * a[i].y + g1[i].y * b[i].y)) +
            ((g0[i].z * a[i].z + g1[i].z * b[i].z) + (g0[i].w * a[i].w + g1[i].w * b[i].w));
    sgr += ((h0[i].x + h1[i].x) + (h0[i].y + h1[i].y)) + ((h0[i].z + h1[i].z) + (h0[i].w + h1[i].w));
    sgxr += ((h0[i].x * b[i].x + h1[i].x * a[i].x) + (h0[i].y * b[i].y + h1[i].y * a[i].y)) +
            ((h0[i].z * b[i].z + h1[i].z * a[i].z) + (h0[i].w * b[i].w + h1[i].w * a[i].w));
  }
  sq = warp_sum(sq), sgk = warp_sum(sgk), sgxk = warp_sum(sgxk), sgr = warp_sum(sgr), sgxr = warp_sum(sgxr);
  const float inv = 1.0f / sqrtf(sq / W + kLnEps);
  const float mgk = sgk / W, mgxk = sgxk * inv / W, mgr = sgr / W, mgxr = sgxr * inv / W;
  // input adjoint of a concat row's element with centred value x and weighted output adjoint g, for row k's / r's statistics
  auto in_k = [&](float g, float x) { return inv * (g - mgk - x * inv * mgxk); };
  auto in_r = [&](float g, float x) { return inv * (g - mgr - x * inv * mgxr); };
  float big_k = 0.f, big_r = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = 128 * i + 4 * lane;
    float4 o = ld4(ie_adj + size_t(k) * D + c);
    o.x += in_k(g0[i].x, a[i].x), o.y += in_k(g0[i].y, a[i].y), o.z += in_k(g0[i].z, a[i].z), o.w += in_k(g0[i].w, a[i].w);
    if (mutual) {
      o.x += in_r(h1[i].x, a[i].x), o.y += in_r(h1[i].y, a[i].y), o.z += in_r(h1[i].z, a[i].z), o.w += in_r(h1[i].w, a[i].w);
      float4 t = ld4(ie_adj + size_t(r) * D + c);
      t.x += in_r(h0[i].x, b[i].x) + in_k(g1[i].x, b[i].x), t.y += in_r(h0[i].y, b[i].y) + in_k(g1[i].y, b[i].y);
      t.z += in_r(h0[i].z, b[i].z) + in_k(g1[i].z, b[i].z), t.w += in_r(h0[i].w, b[i].w) + in_k(g1[i].w, b[i].w);
      st4(edge_adj + size_t(r) * D + c, t);
      big_r = fmaxf(big_r, max4(t));
    }
    st4(edge_adj + size_t(k) * D + c, o);
    big_k = fmaxf(big_k, max4(o));
  }
  if (!mx) return;
  big_k = warp_max(big_k);
  if (mutual) big_r = warp_max(big_r);
  if (lane == 0) {
    mx[k] = __float_as_uint(big_k);
    if (mutual) mx[r] = __float_as_uint(big_r);
  }
}

// send(l, :) = the second half of the norm's input adjoint on live edge l's row: what its partner's rank adds.
__global__ void __launch_bounds__(256) k_concat_norm_remote_bwd(float* __restrict__ send, const float* __restrict__ out_adj,
                                                                const float* __restrict__ oe, const float* __restrict__ w,
                                                                const int* __restrict__ live_packed, int n_live, int D,
                                                                RemoteRows rm) {
  after_previous();
  const int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (l >= n_live) return;
  const int k = live_packed[l], W = 2 * D;
  if (k < 0) {
    for (int d = lane; d < D; d += 32) send[size_t(l) * D + d] = 0.f;
    return;
  }
  const float* b = rm.rows + size_t(l) * D;
  const RowStats sk = concat_stats(oe, b, out_adj, w, k, D, lane);
  for (int d = lane; d < D; d += 32)
    send[size_t(l) * D + d] = sk.inv * (out_adj[size_t(k) * W + D + d] * w[D + d] - sk.mg - (b[d] - sk.mu) * sk.inv * sk.mgx);
}

__global__ void __launch_bounds__(256) k_compress_geometry_bwd(float* __restrict__ x4_adj, const float* __restrict__ g,
                                                               const float* __restrict__ wx, int E, int D, bool add) {
  after_previous();
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (k >= E) return;
  float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
  for (int d = lane; d < D; d += 32) {
    const float gd = g[size_t(k) * D + d];
    const float4 ww = ld4(wx + 4 * d);
    a0 += gd * ww.x, a1 += gd * ww.y, a2 += gd * ww.z, a3 += gd * ww.w;
  }
  a0 = warp_sum(a0), a1 = warp_sum(a1), a2 = warp_sum(a2), a3 = warp_sum(a3);
  if (lane == 0) {
    float4 v = add ? ld4(x4_adj + 4 * size_t(k)) : make_float4(0.f, 0.f, 0.f, 0.f);
    v.x += a0, v.y += a1, v.z += a2, v.w += a3;
    st4(x4_adj + 4 * size_t(k), v);
  }
}

__global__ void k_readout_energy(float* __restrict__ net, double* __restrict__ per_atom, const float* __restrict__ node_pred,
                                 const float* __restrict__ edge_pred, PackedEdges pk, const double* __restrict__ comp,
                                 double scale, bool acc, bool assemble) {
  after_previous();
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (n >= pk.N) return;
  double s = 0.0;
  for (int k = pk.off[n] + lane; k < pk.off[n + 1]; k += 32) s += (double) pk.cut[k] * (double) edge_pred[k];
  s = warp_sum(s);
  if (lane == 0) {
    s += (double) node_pred[n];
    const float v = acc ? (float) ((double) net[n] + s) : (float) s;
    net[n] = v;
    if (assemble) per_atom[n] = n < pk.n_local ? scale * (double) v + comp[pk.atom_species[n]] : 0.0;
  }
}

__global__ void k_readout_seed_bwd(float* __restrict__ out, const float* __restrict__ w, const float* __restrict__ pre,
                                   const float* __restrict__ cut, const int* __restrict__ center, int n_local, int R, int Dh4,
                                   uint32_t* __restrict__ mx) {
  after_previous();
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= size_t(R) * Dh4) return;
  const int r = int(t / Dh4), q = int(t % Dh4);
  float seed;
  if (cut) seed = center[r] < n_local ? cut[r] : 0.f;
  else seed = r < n_local ? 1.f : 0.f;
  const float4 x = reinterpret_cast<const float4*>(pre)[t], ww = reinterpret_cast<const float4*>(w)[q];
  const float4 v = make_float4(seed * ww.x * dsilu_f(x.x), seed * ww.y * dsilu_f(x.y), seed * ww.z * dsilu_f(x.z), seed * ww.w * dsilu_f(x.w));
  reinterpret_cast<float4*>(out)[t] = v;
  raise_row(mx, r, Dh4, max4(v));
}

__global__ void k_cutoff_share(float* __restrict__ cf_adj, const float* __restrict__ cfh, size_t stride, int blocks, const float* __restrict__ cut,
                               int N, int E, int H) {
  after_previous();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= E) return;
  const float cf = cut[k];
  float sum = 0.f;
  if (cf > 0.f)
    for (int b = 0; b < blocks; ++b, cfh += stride) {
      float total = 0.f;
      for (int h = 0; h < H; ++h) total += cfh[size_t(N + k) * H + h];
      sum += total / cf;
    }
  cf_adj[k] = sum;
}

__global__ void k_add_inplace(float* __restrict__ a, const float* __restrict__ b, size_t n) {
  after_previous();
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < n) a[t] += b[t];
}

__global__ void k_message_average(float* __restrict__ ie, const float* __restrict__ oe, const int* __restrict__ rev, int E,
                                  int D4, RemoteRows rm, uint32_t* __restrict__ mx) {
  after_previous();
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= size_t(E) * D4) return;
  const int k = int(t / D4), q = int(t % D4);
  float4 x = reinterpret_cast<float4*>(ie)[t];
  const float* pr = partner_row(oe, rev, rm, k, 4 * D4);
  const float4 y = pr ? ld4(pr + 4 * q) : make_float4(0, 0, 0, 0);
  x = make_float4(0.5f * (x.x + y.x), 0.5f * (x.y + y.y), 0.5f * (x.z + y.z), 0.5f * (x.w + y.w));
  reinterpret_cast<float4*>(ie)[t] = x;
  raise_row(mx, k, D4, max4(x));
}

// The adjoint of message_average: ie_adj_out(k) = 0.5 ie_adj_in(k); oe_adj(k) += 0.5 ie_adj_in(rev k).
__global__ void k_message_average_bwd(float* __restrict__ ie_out, float* __restrict__ oe_adj, const float* __restrict__ ie_in,
                                      const int* __restrict__ rev, int E, int D4, RemoteRows rm) {
  after_previous();
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= size_t(E) * D4) return;
  const int k = int(t / D4), q = int(t % D4);
  const float4 x = reinterpret_cast<const float4*>(ie_in)[t];
  float4 o = reinterpret_cast<float4*>(oe_adj)[t];
  const float* pr = partner_row(ie_in, rev, rm, k, 4 * D4);  // the partner edge's adjoint row, here or from its rank
  if (pr) {
    const float4 y = ld4(pr + 4 * q);
    o.x += 0.5f * y.x, o.y += 0.5f * y.y, o.z += 0.5f * y.z, o.w += 0.5f * y.w;
  }
  reinterpret_cast<float4*>(oe_adj)[t] = o;
  reinterpret_cast<float4*>(ie_out)[t] = make_float4(0.5f * x.x, 0.5f * x.y, 0.5f * x.z, 0.5f * x.w);
}

// The smooth cutoff's derivative in the distance, in float like the factor itself
// (bump_ddist / cosine_ddist, src/forces.cpp:22-35).
__device__ inline double cutoff_ddist(double d, double rc, double w, int kind) {
  const float pi = (float) 3.14159265358979323846;
  const float x = (float) ((d - (rc - w)) / w);
  if (x <= 0.f || x >= 1.f) return 0.0;
  if (kind == 0) {
    const float si = sinf(pi * x);
    const float t = tanhf(cosf(pi * x) / si);
    const float du = (-pi / (si * si)) / (float) w;
    return 0.5 * (1.0 - (double) (t * t)) * (double) du;
  }
  return 0.5 * (double) (-pi * sinf(pi * x)) / w;
}

// pc_adj, unless null, receives the adjoint of the edge's own cutoff (an adaptive cutoff): the factor depends on
// d - rc, so it is minus the distance's share (src/forces.cpp:372-377).
__global__ void k_edge_grad(double* __restrict__ grad, PackedEdges pk, const float* __restrict__ x4_adj,
                            const float* __restrict__ cutoff_adj, const float* __restrict__ cf_adj, CutoffSpec cs,
                            double* __restrict__ pc_adj) {
  after_previous();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= pk.E) return;
  if (pc_adj && k >= pk.off[pk.N]) {  // a capacity's dead row
    pc_adj[k] = 0.0;
    for (int c = 0; c < 3; ++c) grad[3 * size_t(k) + c] = 0.0;
    return;
  }
  const bool own = pk.center[k] < pk.n_local;
  const double cutoff_total = (own ? (double) cutoff_adj[k] : 0.0) + (double) cf_adj[k];
  const double d = pk.dist[k];
  const double dcut_dd = cutoff_ddist(d, pk.rc ? pk.rc[k] : cs.cutoff, cs.width, cs.kind);
  if (pc_adj) pc_adj[k] = -cutoff_total * dcut_dd;
  const double dist_adj = (double) x4_adj[4 * size_t(k) + 3] + cutoff_total * dcut_dd;
  const double invd = d > 0.0 ? 1.0 / d : 0.0;
  for (int c = 0; c < 3; ++c) grad[3 * size_t(k) + c] = (double) x4_adj[4 * size_t(k) + c] + dist_adj * pk.vec[3 * size_t(k) + c] * invd;
}

// One warp per atom: F(i) = scale sum_k [g(k) - g(rev k)], W(i) = scale sum_k v (x) g, lanes striding
// the atom's edges and combining in a fixed tree.
__global__ void __launch_bounds__(256) k_fold_forces(ForceOut out, PackedEdges pk, double scale) {
  after_previous();
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= pk.n_atoms) return;
  double f[3] = {0, 0, 0}, w[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (i < pk.N)
    for (int k = pk.off[i] + lane; k < pk.off[i + 1]; k += 32) {
      const double* g = out.edge_grad + 3 * size_t(k);
      const double* v = pk.vec + 3 * size_t(k);
      const int r = pk.reverse[k];
      for (int c = 0; c < 3; ++c) f[c] += g[c] - (r >= 0 ? out.edge_grad[3 * size_t(r) + c] : 0.0);
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) w[a * 3 + b] += v[a] * g[b];
    }
  for (int c = 0; c < 3; ++c) f[c] = warp_sum(f[c]);
  for (int t = 0; t < 9; ++t) w[t] = warp_sum(w[t]);
  if (lane == 0) {
    for (int c = 0; c < 3; ++c) out.forces[3 * size_t(i) + c] = scale * f[c];
    for (int t = 0; t < 9; ++t) out.vir_atom[9 * size_t(i) + t] = scale * w[t];
  }
}

// Structure b's energy and, unless w6 is null, its virial in Voigt's order from the atoms' 3 x 3: the ordered sum over its atoms, of both
// elements of a symmetric pair where there are two. A block per sum, whose warps' parts are added in order: a warp alone takes 12 us
// for 1728 atoms, one trip to L2 after another. All of them in one launch (three launches before).
__global__ void __launch_bounds__(256) k_struct_sums(double* __restrict__ energy, double* __restrict__ w6, const double* __restrict__ per_atom,
                                                     const double* __restrict__ vir_atom, const int* __restrict__ soff) {
  after_previous();
  __shared__ double part[2][8];
  const int T = w6 ? 7 : 1, b = blockIdx.x / T, t = blockIdx.x % T, end = soff[b + 1];
  const bool is_energy = t + 1 == T;
  constexpr int first[6] = {0, 4, 8, 1, 2, 5}, second[6] = {0, 4, 8, 3, 6, 7};
  const double *x = per_atom, *y = per_atom;
  int ld = 1;
  if (!is_energy) {
    ld = 9;
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (i == t) x = vir_atom + first[i], y = vir_atom + second[i];
  }
  const bool pair = x != y;
  double s = 0.0, r = 0.0;
#pragma unroll 4
  for (int a = soff[b] + threadIdx.x; a < end; a += 256) {
    s += x[size_t(a) * ld];
    if (pair) r += y[size_t(a) * ld];
  }
  s = warp_sum(s), r = warp_sum(r);
  if (threadIdx.x % 32 == 0) part[0][threadIdx.x / 32] = s, part[1][threadIdx.x / 32] = r;
  __syncthreads();
  if (threadIdx.x) return;
  for (int w = 1; w < 8; ++w) s += part[0][w], r += part[1][w];
  if (is_energy) energy[b] = s;
  else w6[6 * b + t] = pair ? 0.5 * (s + r) : s;
}

inline unsigned blocks_for(size_t n, int per) { return (unsigned) ((n + per - 1) / per); }

}  // namespace

void gather_rows(Stream& st, float* out, const float* table, const int* idx, int R, int D, uint32_t* mx) {
  gather_rows_two(st, out, table, idx, R, D, mx, nullptr, nullptr, nullptr, 0, 4);
}
void gather_rows_two(Stream& st, float* out, const float* table, const int* idx, int R, int D, uint32_t* mx, float* out2, const float* table2,
                     const int* idx2, int R2, int D2) {
  if (R == 0 && R2 == 0) return;
  const ProfScope ps(st, PC_GATHER, 0.0, 8.0 * (double(R) * D + double(R2) * D2));
  const unsigned blocks0 = blocks_for(size_t(R) * (D / 4), 256);
  launch(st, k_gather_rows, blocks0 + blocks_for(size_t(R2) * (D2 / 4), 256), 256, 0, Lookup{out, table, idx, mx, R, D / 4},
         Lookup{out2, table2, idx2, nullptr, R2, D2 / 4}, int(blocks0));
  PETB_LAUNCH_CHECK(st);
}

void compress0(Stream& st, float* out, float* pre, const float* b, const float* tab, const float* wx, const PackedEdges& pk,
               int D, uint32_t* mx) {
  if (pk.E == 0) return;
  const ProfScope ps(st, PC_ELEMENTWISE, 12.0 * double(pk.E) * D, 8.0 * double(pk.E) * D);
  GemmArgs p;
  p.M = pk.E, p.N = D, p.C = out, p.ldc = D, p.pre = pre, p.ldp = D, p.bias = b, p.tab = tab, p.wx = wx, p.sp = pk.species;
  p.vec = pk.vec, p.dist = pk.dist, p.c_max = mx, p.epi = EPI_COMPRESS;
  const int rows = pk.E < 16384 ? 1 : 8;  // (few rows: all SMs)
  launch(st, k_compress0, blocks_for(size_t(cdiv(pk.E, rows)) * (D / 4), 256), 256, 0, p, rows);
  PETB_LAUNCH_CHECK(st);
}

void norm_fwd(Stream& st, float* out, float* in, const float* add, const float* w, const float* bias, int R, int D, uint32_t* mx) {
  if (R == 0) return;
  const ProfScope ps(st, PC_NORM, 6.0 * double(R) * D, (add ? 16.0 : 8.0) * double(R) * D);
  const unsigned blocks = blocks_for(size_t(R) * 32, 256);
  switch (D) {  // whole rows in registers for the usual widths
    case 128: launch(st, k_norm_fwd_v<1>, blocks, 256, 0, out, in, add, w, bias, R, mx); break;
    case 256: launch(st, k_norm_fwd_v<2>, blocks, 256, 0, out, in, add, w, bias, R, mx); break;
    case 512: launch(st, k_norm_fwd_v<4>, blocks, 256, 0, out, in, add, w, bias, R, mx); break;
    case 1024: launch(st, k_norm_fwd_v<8>, blocks, 256, 0, out, in, add, w, bias, R, mx); break;
    default: launch(st, k_norm_fwd, blocks, 256, 0, out, in, add, w, bias, R, D, mx);
  }
  PETB_LAUNCH_CHECK(st);
}

void gather_live(Stream& st, float* out, const float* src, int ld, int col0, const int* live_packed, int n_live, int D) {
  if (n_live == 0) return;
  const ProfScope ps(st, PC_GATHER, 0.0, 8.0 * double(n_live) * D);
  launch(st, k_gather_live, blocks_for(size_t(n_live) * (D / 4), 256), 256, 0, out, src, ld, col0, live_packed, n_live, D / 4);
  PETB_LAUNCH_CHECK(st);
}

void concat_norm_fwd(Stream& st, float* out, const float* oe, const int* rev, float* ie, const float* w, const float* bias,
                     int E, int D, RemoteRows remote, uint32_t* mx) {
  if (E == 0) return;
  const ProfScope ps(st, PC_NORM, 12.0 * double(E) * D, 24.0 * double(E) * D);
  launch(st, k_concat_norm_fwd, blocks_for(size_t(E) * 32, 256), 256, 0, out, oe, rev, ie, w, bias, E, D, remote, mx);
  PETB_LAUNCH_CHECK(st);
}

void norm_bwd(Stream& st, float* in_adj, const float* out_adj, const float* in, const float* w, bool layernorm, int R, int D,
              int acc_row0, float* also, uint32_t* mx) {
  if (R == 0) return;
  const ProfScope ps(st, PC_NORM, 10.0 * double(R) * D, (acc_row0 < R ? 16.0 : 12.0) * double(R) * D);
  const unsigned blocks = blocks_for(size_t(R) * 32, 256);
  switch (D) {
    case 128: launch(st, k_norm_bwd_v<1>, blocks, 256, 0, in_adj, out_adj, in, w, layernorm, R, acc_row0, also, mx); break;
    case 256: launch(st, k_norm_bwd_v<2>, blocks, 256, 0, in_adj, out_adj, in, w, layernorm, R, acc_row0, also, mx); break;
    case 512: launch(st, k_norm_bwd_v<4>, blocks, 256, 0, in_adj, out_adj, in, w, layernorm, R, acc_row0, also, mx); break;
    case 1024: launch(st, k_norm_bwd_v<8>, blocks, 256, 0, in_adj, out_adj, in, w, layernorm, R, acc_row0, also, mx); break;
    default: launch(st, k_norm_bwd, blocks, 256, 0, in_adj, out_adj, in, w, layernorm, R, D, acc_row0, also, mx);
  }
  PETB_LAUNCH_CHECK(st);
}

void norm_bwd_two(Stream& st, float* n_adj, const float* n_out_adj, const float* n_in, const float* n_w, int N, int Dn, uint32_t* n_mx,
                  float* e_adj, const float* e_out_adj, const float* e_in, const float* e_w, int E, int D, uint32_t* e_mx) {
  if (N == 0 && E == 0) return;
  if (Dn > 2048 || (D != 128 && D != 256 && D != 512)) {
    norm_bwd(st, e_adj, e_out_adj, e_in, e_w, false, E, D, 0, nullptr, e_mx);
    return norm_bwd(st, n_adj, n_out_adj, n_in, n_w, false, N, Dn, 0, nullptr, n_mx);
  }
  const double values = double(N) * Dn + double(E) * D;
  const ProfScope ps(st, PC_NORM, 10.0 * values, 16.0 * values);
  const NormBwdRows n{n_adj, n_out_adj, n_in, n_w, n_mx, N, Dn}, e{e_adj, e_out_adj, e_in, e_w, e_mx, E, D};
  const auto kernel = D == 128 ? k_norm_bwd_two<1> : D == 256 ? k_norm_bwd_two<2> : k_norm_bwd_two<4>;
  launch(st, kernel, size_t(N) + blocks_for(E, 8), 256, 0, n, e);
  PETB_LAUNCH_CHECK(st);
}

void concat_norm_bwd(Stream& st, float* edge_adj, const float* out_adj, const float* oe, const int* rev, const float* ie_adj,
                     const float* w, int E, int D, RemoteRows remote, const float* remote_adj, uint32_t* mx) {
  if (E == 0) return;
  const ProfScope ps(st, PC_NORM, 20.0 * double(E) * D, 24.0 * double(E) * D);
  const auto grid = blocks_for(size_t(E) * 32, 256);
  const bool one_rank = !remote.of && !remote_adj;
  if (one_rank && D == 128)
    launch(st, k_concat_norm_bwd_pair<1>, grid, 256, 0, edge_adj, out_adj, oe, rev, ie_adj, w, E, mx);
  else if (one_rank && D == 256)
    launch(st, k_concat_norm_bwd_pair<2>, grid, 256, 0, edge_adj, out_adj, oe, rev, ie_adj, w, E, mx);
  else if (one_rank && D == 512)
    launch(st, k_concat_norm_bwd_pair<4>, grid, 256, 0, edge_adj, out_adj, oe, rev, ie_adj, w, E, mx);
  else
    launch(st, k_concat_norm_bwd, grid, 256, 0, edge_adj, out_adj, oe, rev, ie_adj, w, E, D, remote, remote_adj, mx);
  PETB_LAUNCH_CHECK(st);
}

void concat_norm_remote_bwd(Stream& st, float* send, const float* out_adj, const float* oe, const float* w,
                            const int* live_packed, int n_live, int D, RemoteRows remote) {
  if (n_live == 0) return;
  const ProfScope ps(st, PC_NORM, 20.0 * double(n_live) * D, 16.0 * double(n_live) * D);
  launch(st, k_concat_norm_remote_bwd, blocks_for(size_t(n_live) * 32, 256), 256, 0, send, out_adj, oe, w, live_packed, n_live, D,
                                                                                  remote);
  PETB_LAUNCH_CHECK(st);
}

void compress_geometry_bwd(Stream& st, float* x4_adj, const float* g, const float* wx, int E, int D, bool add) {
  if (E == 0) return;
  const ProfScope ps(st, PC_ELEMENTWISE, 8.0 * double(E) * D, 4.0 * double(E) * D);
  launch(st, k_compress_geometry_bwd, blocks_for(size_t(E) * 32, 256), 256, 0, x4_adj, g, wx, E, D, add);
  PETB_LAUNCH_CHECK(st);
}

void readout_energy(Stream& st, float* net, double* per_atom, const float* node_pred, const float* edge_pred,
                    const PackedEdges& pk, const double* composition, double scale, bool acc, bool assemble) {
  if (pk.N == 0) return;
  const ProfScope ps(st, PC_GATHER, 2.0 * pk.E, 8.0 * double(pk.E) + 16.0 * pk.N);
  launch(st, k_readout_energy, blocks_for(size_t(pk.N) * 32, 256), 256, 0, net, per_atom, node_pred, edge_pred, pk, composition,
                                                                        scale, acc, assemble);
  PETB_LAUNCH_CHECK(st);
}

void readout_seed_bwd(Stream& st, float* out, const float* w, const float* pre, const float* cut, const int* center,
                      int n_local, int R, int Dh, uint32_t* mx) {
  if (R == 0) return;
  const ProfScope ps(st, PC_ELEMENTWISE, 8.0 * double(R) * Dh, 8.0 * double(R) * Dh);
  launch(st, k_readout_seed_bwd, blocks_for(size_t(R) * (Dh / 4), 256), 256, 0, out, w, pre, cut, center, n_local, R, Dh / 4, mx);
  PETB_LAUNCH_CHECK(st);
}

void cutoff_share(Stream& st, float* cf_adj, const float* cfh, size_t stride, int blocks, const float* cut, int N, int E, int H) {
  if (E == 0) return;
  const ProfScope ps(st, PC_ELEMENTWISE, double(E) * H * blocks, 4.0 * double(E) * (H * blocks + 2));
  launch(st, k_cutoff_share, blocks_for(E, 256), 256, 0, cf_adj, cfh, stride, blocks, cut, N, E, H);
  PETB_LAUNCH_CHECK(st);
}

void add_inplace(Stream& st, float* a, const float* b, size_t n) {
  if (n == 0) return;
  const ProfScope ps(st, PC_ELEMENTWISE, double(n), 12.0 * double(n));
  launch(st, k_add_inplace, blocks_for(n, 256), 256, 0, a, b, n);
  PETB_LAUNCH_CHECK(st);
}

void message_average(Stream& st, float* ie, const float* oe, const int* rev, int E, int D, RemoteRows remote,
                     uint32_t* mx) {
  if (E == 0) return;
  const ProfScope ps(st, PC_GATHER, 2.0 * double(E) * D, 12.0 * double(E) * D);
  launch(st, k_message_average, blocks_for(size_t(E) * (D / 4), 256), 256, 0, ie, oe, rev, E, D / 4, remote, mx);
  PETB_LAUNCH_CHECK(st);
}

void message_average_bwd(Stream& st, float* ie_adj_out, float* oe_adj, const float* ie_adj_in, const int* rev, int E, int D,
                         RemoteRows remote_adj) {
  if (E == 0) return;
  const ProfScope ps(st, PC_GATHER, 2.0 * double(E) * D, 20.0 * double(E) * D);
  launch(st, k_message_average_bwd, blocks_for(size_t(E) * (D / 4), 256), 256, 0, ie_adj_out, oe_adj, ie_adj_in, rev, E, D / 4,
                                                                              remote_adj);
  PETB_LAUNCH_CHECK(st);
}

void forces_and_virial(Stream& st, Arena& arena, ForceOut& out, const PackedEdges& pk, const float* x4_adj, const float* cutoff_adj,
                       const float* cf_adj, const CutoffSpec& cs, double scale, double* energy, const double* per_atom) {
  const ProfScope ps(st, PC_FORCES, 40.0 * pk.E, 100.0 * double(pk.E) + 96.0 * pk.n_atoms);
  double* pc_adj = pk.adaptive.acut ? arena.alloc<double>(pk.E > 0 ? pk.E : 1) : nullptr;
  if (pk.E > 0) {
    launch(st, k_edge_grad, blocks_for(pk.E, 256), 256, 0, out.edge_grad, pk, x4_adj, cutoff_adj, cf_adj, cs, pc_adj);
    PETB_LAUNCH_CHECK(st);
  }
  if (pk.n_atoms > 0) {
    launch(st, k_fold_forces, blocks_for(size_t(pk.n_atoms) * 32, 256), 256, 0, out, pk, scale);
    PETB_LAUNCH_CHECK(st);
  }
  // the adaptive cutoff's share, folded over the raw list, before the per-structure sums
  if (pc_adj) adaptive_backward(st, arena, pk, cs, pc_adj, scale, out.forces, out.vir_atom, &out.adaptive_gmag);
  structure_sums(st, energy, out.vir6, per_atom, out.vir_atom, pk.soff, pk.B);
}

void structure_sums(Stream& st, double* energy, double* vir6, const double* per_atom, const double* vir_atom, const int* soff, int B) {
  launch(st, k_struct_sums, size_t(B) * (vir6 ? 7 : 1), 256, 0, energy, vir6, per_atom, vir_atom, soff);
  PETB_LAUNCH_CHECK(st);
}

}  // namespace petb
