// The tensor-core GEMM: tcgen05.mma kind::f16 with TMA-fed shared-memory tiles and the accumulators in tensor memory
// (sm_100a). See gemm.h for the interface, the operand formats and the epilogues.
//
// A persistent kernel, one CTA per SM, each walking 128 x BN tiles of C = A . B^T (A [M,K] fp32, B [N,K] a packed
// weight) in an N-fastest order so that CTAs running side by side share their A rows in L2. K goes by steps of 32
// columns (FMT_TF32X2: 16). Roles, by warp:
//   warp 0      producer of A: one lane issues TMA loads of 128 x 32 fp32 slabs (128-byte rows, 128-byte swizzle) into a
//               ring of slots; warp 2 the same for B's tiles, which arrive as 16-bit parts;
//   warps 12-15 converter: a lane takes one row's 128 bytes out of a landed slot, scales and splits it and writes the
//               parts back into the same 128 bytes (64 bytes a part; FMT_F16X3's third part into a tile of its own): a slot costs
//               no second copy of A. The fp32 activations are read from memory once;
//   warp 1      issuer: one lane issues the products (M = 128, N = BN, K = 16 each) into one of TWO accumulators in
//               tensor memory, small terms first, and frees the step's slots with one tcgen05.commit;
//   warps 4-11  epilogue: tcgen05.ld the accumulator (a thread owns a row, a warp pair splits the columns), undo the
//               two rows' scales, and work through 32 x 32 chunks in shared memory: what the epilogue reads (a
//               residual, a saved pre-activation) is brought there by TMA a chunk ahead, what it writes leaves by TMA. The
//               accumulator is handed back as soon as it has been read.
// FMT_F16X3 fills both accumulators for one tile (the exact h.h sum, and the small products); the epilogue warps add the two into
// registers, rounding once, and hand them back before they start on the chunks. The tensor core truncates its fp32
// accumulator at every instruction: on sums with more bits than it keeps that is a bias toward zero which adds up over K
// and over a network (two truncations per 32 columns were enough to move energies by 1e-6). The h.h sums have no such
// bits, and the small products' truncations are 2^-8 of what they would be there (where most values have a leading part:
// FMT_F16X3_FULL in gemm.h). setmaxnreg moves the registers the sums
// take from the producers' and converters' warp groups.
// Large GEMMs in the formats of several parts run on pairs of CTAs (cta_group::2): 256 x 256 tiles, each CTA with 128 rows of
// A and half of the weight's tile in its shared memory, its own converter and epilogue, one issuer for both. A CTA's
// converter tells the issuer that a step's operands are complete by an arrival on its barrier across the cluster, without a
// cluster-scope release: that one (or an acquire on the waiting side) costs 2500 clocks a step. The converter's own writes
// are ordered by the proxy fence before the arrival, and nothing but the tensor core reads them.
//
// The other tiles (Tile::TA: not the pairs, not the tf32 formats, and with parts to spare in tensor memory) keep A's parts in
// tensor memory instead: two groups of four converter warps (12-19) take a slab out of shared memory, which frees its slot at
// once, and store the parts with tcgen05.st as the A operand of the products, 16 columns a part. That takes A's second trip
// through shared memory and the proxy fence out of a step. Every role asks for its next step's barrier (mbar_test) before it
// works on this step's: an answer takes 150 clocks, a third of a step of a narrow tile.
// Where a GEMM has few tiles (the atoms' rows), a step's chain of barriers bounds it, not any unit's rate. 648 rows of a
// recorded pass, FMT_F16X2: N 1024 K 4096 64.7 us -> 47.1, N 256 K 1024 18.3 -> 14.2, N 1024 K 256 7.7 -> 7.1; FMT_F16X3,
// 21 rows, N 512 K 2048: 35.0 -> 27.4.
//
// What bounds the large ones: no unit is at its rate. Counters of 122138 x 256 x 256 in three, two and one parts: tensor pipe
// active 69, 53 and 21 % of the active cycles, SM memory throughput 60, 45 and 18 %, DRAM 29, 43 and 50 %, issue slots 50, 39 and
// 42 %; in a fifth of the elapsed cycles no SM is active. The most work falls on the shared-memory data path (one 128-byte
// wavefront per clock for TMA traffic, the tensor core's operand reads, the converter and the epilogue). Wavefronts per 8
// columns of K of a 128 x 256 tile, K = 256, by count: FMT_F16X2 operand reads 144, fills 96, converter 64, epilogue 64-128 =
// about 370-430 against 192 clocks of MMA; FMT_F16X3 288, 128, 80, 64-128 = about 560-620 against 384. A step's chain of
// barriers, and an epilogue that has the one accumulator of 256 columns to itself, leave each of them idle in between.
// No TMA load here uses cluster multicast. Every wait is bounded: a wait that runs out sets an error word the host checks,
// every role then leaves its loop, and the CTA still reaches its tensor-memory release.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "epilogue.cuh"
#include "gemm_tc.h"
#include "tcgen05.cuh"

namespace petb {

namespace {

constexpr int TBM = 128;  // rows of a tile
constexpr int kEpiWarp0 = 4, kEpiWarps = 8, kConvWarp0 = 12;

// ---- the fp16 formats' scales --------------------------------------------------------------
// The power of two that brings a row whose largest magnitude has these bits to [2^14, 2^15), and its inverse.
// Rows below 2^-112 are taken as that, which keeps both normal numbers.
__device__ __forceinline__ uint32_t scale_exponent(uint32_t max_bits) { return max(max_bits >> 23, 15u); }
__device__ __forceinline__ float scale_of(uint32_t max_bits) { return __uint_as_float((268u - scale_exponent(max_bits)) << 23); }
__device__ __forceinline__ float unscale_of(uint32_t max_bits) { return __uint_as_float((scale_exponent(max_bits) - 14u) << 23); }

__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t pack_f16(float x, float y) {
  const __half2 v = __floats2half2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_f16(uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }

// Two neighbouring values into their parts. `s` is the row's scale (fp16 formats).
template <int FMT>
__device__ __forceinline__ void split2(float x, float y, float s, uint32_t& h, uint32_t& m, uint32_t& l) {
  if (three_parts(FMT)) {
    constexpr float kGrid = 3221225472.f;  // 1.5 2^31: adding it rounds to a multiple of 2^8
    x *= s, y *= s;
    const float xh = (x + kGrid) - kGrid, yh = (y + kGrid) - kGrid;
    h = pack_f16(xh, yh);  // exact
    x -= xh, y -= yh;      // exact
    m = pack_f16(x, y);
    const float2 a = unpack_f16(m);
    l = pack_f16(x - a.x, y - a.y);
  } else if (FMT == FMT_F16X2) {
    x *= s, y *= s;
    h = pack_f16(x, y);
    const float2 a = unpack_f16(h);
    m = pack_f16(x - a.x, y - a.y);
  } else if (FMT == FMT_F16) {  // exact but for values below 2^-28 of the row's largest
    h = pack_f16(__uint_as_float(__float_as_uint(x) & 0xFFFFE000u) * s, __uint_as_float(__float_as_uint(y) & 0xFFFFE000u) * s);
  } else {
    h = pack_bf16(x, y);
  }
}

// The low part of the tf32 split. The tensor core reads the top 19 bits of an fp32 operand (sign, exponent, 10 mantissa
// bits), so h(x) is x truncated; x - h(x) is exact and has up to 13 significant bits, of which the tensor core would again
// keep the top 11 by truncation. Adding half of the last kept bit makes that a rounding to nearest.
__device__ __forceinline__ float tf32_low(float x) {
  return __uint_as_float(__float_as_uint(x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u)) + 0x1000u);
}

template <int BN, int FMT, bool PAIR>
struct Tile {
  static constexpr bool X3 = three_parts(FMT), kFull = FMT == FMT_F16X3_FULL, X2 = FMT == FMT_F16X2, T2 = FMT == FMT_TF32X2, T1 = FMT == FMT_TF32;
  static constexpr bool kScaled = scales_rows(FMT);
  static constexpr int BK = T2 ? 16 : 32;                                   // columns of K of a step
  // A's parts in tensor memory, where the accumulators leave room for them.
  static constexpr bool TA = !PAIR && !T1 && !T2 && (X2 || BN <= 128);
  static constexpr int kParts = X3 ? 3 : X2 ? 2 : 1;
  static constexpr int kSlab = TBM * BK * 4;                                // A as it lands
  static constexpr int kA = kSlab + ((X3 && !TA) || T2 ? TBM * 64 : 0);     // the fp32 slab, then its parts; l behind it
  static constexpr int kRowsB = PAIR ? BN / 2 : BN;                         // of B's tile, in this CTA
  static constexpr int kB = kRowsB * (X3 ? 192 : X2 || T2 || T1 ? 128 : 64);          // [h | m] or [h | l] rows of 128 bytes (then l), or rows of 64
  // An epilogue warp's two buffers of 32 rows x kWide columns; half as wide where the rings need the room.
  static constexpr int kWide = X3 ? 16 : 32;
  static constexpr int kBuf = 32 * kWide * 4;
  static constexpr int kEpi = kEpiWarps * 2 * kBuf;
  static constexpr int kBars = 640;
  // Slots: as many as shared memory has room for beside the epilogue's buffers, at most eight of each; of A, whose bytes come
  // from HBM, no fewer than of B, whose bytes sit in L2; of A an even number, for the converter's groups.
  static constexpr int kRows = 2 * TBM * 4;  // a tile's rows' sums of squares, by group of the converter
  static constexpr int kRoom = 227 * 1024 - kEpi - 1024 - kBars - kRows;
  static constexpr int least(int a, int b) { return a < b ? a : b; }
  static constexpr int slots_a(int nb) { return least(8, (kRoom - nb * kB) / kA); }
  static constexpr int kBoth = least(8, kRoom / (kA + kB));
  static constexpr bool kTrade = slots_a(kBoth) % 2 != 0 && slots_a(kBoth - 1) % 2 == 0;  // one of B's for one more of A's
  // TA: A's slots are free as soon as they are read, four will do; B's no more than the steps of A's parts (NT).
  static constexpr int kBesideFour = least(X3 ? 5 : 8, (kRoom - 4 * kA) / kB);
  static constexpr int NB = TA ? kBesideFour : least(kTrade ? kBoth - 1 : kBoth, slots_a(kTrade ? kBoth - 1 : kBoth) / 2 * 2);
  static constexpr int NA = slots_a(TA ? NB : kTrade ? kBoth - 1 : kBoth) / 2 * 2;
  // The converter's warps work in groups on slots of their own: a slot takes a warp about a thousand clocks however few
  // instructions its rows need (the wait, the loads, the fence), so two or four of them have to be under way at once. A
  // slot always falls to the same group (NA a multiple of the groups): a group that met a slot's barrier only every other
  // round could take the round before last for the one it waits for.
  // TA: a warp reaches only its quarter of tensor memory's lanes, so a group is four warps, and there are two of them.
  static constexpr int kGroups = !TA && NA % 4 == 0 && NA >= 8 ? 4 : 2;
  static constexpr int kRings = NA * kA + NB * kB;
  static constexpr int kTotal = kRings + kEpi + 1024 /*alignment slack*/ + kBars + kRows;
  static constexpr int kThreads = TA ? 640 : 512;
  // registers of the tile's sums that an epilogue thread keeps over the steps (FMT_F16X3)
  static constexpr int kSums = X3 ? BN / 2 : 1;
  // accumulators in tensor memory: a tile takes one (two in FMT_F16X3), and while it is being read the next tile fills the
  // others, where there are others
  static constexpr int kAccs = X3 ? 2 : 1, kTurns = (TA ? 384 : 512) / (kAccs * BN) >= 2 ? 2 : 1, kColumns = TA ? 512 : kTurns * kAccs * BN;
  // TA: the steps of A's parts behind them, 16 columns a part; ND barriers for the steps' ends, no fewer than any ring's slots
  static constexpr int kPartsAt = kTurns * kAccs * BN, NT = least(8, (512 - kPartsAt) / (16 * kParts)), ND = TA ? 8 : NA;
  static constexpr int NS = TA ? NT : NA;  // `ready` barriers
  // Steps whose products go into one accumulator. FMT_F16X3's h.h products sum exactly over 1024 columns of K; up to 4096 a
  // longer K goes in four pieces, one for each of four CTAs that share a tile (SPLIT).
  static __device__ int drain(int K) { return !X3 ? 1 << 30 : K > 1024 && K <= 4096 ? (K + 127) / 128 : 1024 / BK; }
  // 40 + 2 x 192 + 88 registers a thread over the warp groups are the 4 x 128 of the launch; 48 + 2 x 136 + 2 x 80 the 5 x 96
  static constexpr bool kMoveRegs = TA || (X3 && BN >= 128);
  static constexpr int kRegsProd = TA ? 48 : 40, kRegsEpi = TA ? 136 : 192, kRegsConv = TA ? 80 : 88;
  static_assert(!T1 || !PAIR, "FMT_TF32 has no converter to tell the other CTA's issuer that a slab has landed");
  static_assert(kRings >= TBM * BN * 4, "the shared sums of a split tile");
  static_assert((TA || NA >= NB) && NA >= 2 && NB >= 2 && NA % kGroups == 0, "the slots");
  static_assert(!TA || (NT >= NB && NT <= ND), "the slots");
  static_assert((2 * NA + NS + ND + 6 + 2 * kEpiWarps) * 8 + 8 <= kBars, "the barriers");
};

// Rows of A's TMA box: a matrix of few rows has only its own fetched (a box's rows past the matrix cost as much as others).
__host__ __device__ constexpr int box_rows(int M) { return M >= TBM ? TBM : (M + 31) / 32 * 32; }

// ---- the epilogue ---------------------------------------------------------------------------

constexpr bool reads(int epi) { return epi == EPI_PLAIN || epi == EPI_SILU_BWD || epi == EPI_SWIGLU_BWD; }     // a chunk of `res` or `pre`
constexpr bool writes_two(int epi) { return epi == EPI_SILU || epi == EPI_SWIGLU || epi == EPI_COMPRESS; }     // `pre` beside C

// The lines of its next tile an epilogue warp will read, asked of HBM while it waits for the tile's accumulator: the TMA
// loads of the chunks then find them in L2. A lane asks for its row.
template <int EPI>
__device__ __forceinline__ void epilogue_prefetch(const GemmArgs& p, int row, int col0, int ncols) {
  if (row >= p.M) return;
  const float* base = EPI == EPI_PLAIN ? p.res : p.pre;
  const int wide = EPI == EPI_SWIGLU_BWD ? 2 : 1;
  if (!base || (EPI == EPI_PLAIN && row < p.res_row0)) return;
  if (col0 + ncols > p.N) ncols = p.N - col0;
  const float* r = base + size_t(row) * (EPI == EPI_PLAIN ? p.ldr : p.ldp) + size_t(wide) * col0;
  for (int c = 0; c < wide * ncols; c += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(r + c));
}

// What the compress epilogue reads of its row.
struct RowTerms {
  const float* tab;    // the species' row of the table
  float e0, e1, e2, e3;  // the edge's (v, |v|) in float
};

// `n` accumulators v of one row from column col on (n a multiple of four, N too): `in` is the chunk the epilogue reads, `out` what
// goes to C and `pre` what goes to the saved pre-activation. SWIGLU: n / 2 outputs; SWIGLU_BWD: 2 n inputs and outputs.
template <int EPI, int n>
__device__ __forceinline__ void epilogue_row(const GemmArgs& p, int row, int col, const RowTerms& rt, float* v, bool has_in, const float* in,
                                             float* out, float* pre) {
  if (EPI == EPI_PLAIN || EPI == EPI_SILU || EPI == EPI_SWIGLU || EPI == EPI_COMPRESS) {
    if (p.bias) {
#pragma unroll
      for (int j = 0; j < n; j += 4)
        if (col + j < p.N) {
          const float4 b = ld4(p.bias + col + j);
          v[j] += b.x, v[j + 1] += b.y, v[j + 2] += b.z, v[j + 3] += b.w;
        }
    }
  }
  if (EPI == EPI_COMPRESS) {
#pragma unroll
    for (int j = 0; j < n; j += 4)
      if (col + j < p.N) {
        const float4 t4 = ld4(rt.tab + col + j);
        const float t[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 w = ld4(p.wx + size_t(col + j + i) * 4);
          v[j + i] = v[j + i] + t[i] + w.x * rt.e0 + w.y * rt.e1 + w.z * rt.e2 + w.w * rt.e3;
        }
      }
  }
  if (EPI == EPI_PLAIN) {
    const bool add = has_in && row >= p.res_row0;
#pragma unroll
    for (int j = 0; j < n; ++j) out[j] = add ? v[j] + in[j] : v[j];
  } else if (EPI == EPI_SILU || EPI == EPI_COMPRESS) {
#pragma unroll
    for (int j = 0; j < n; ++j) pre[j] = v[j], out[j] = silu_f(v[j]);
  } else if (EPI == EPI_SWIGLU) {
#pragma unroll
    for (int j = 0; j < n; ++j) pre[j] = v[j];
#pragma unroll
    for (int j = 0; j < n; j += 2) out[j / 2] = v[j] * sigmoid_f(v[j + 1]);
  } else if (EPI == EPI_SILU_BWD) {
#pragma unroll
    for (int j = 0; j < n; ++j) out[j] = v[j] * dsilu_f(in[j]);
  } else if (EPI == EPI_SWIGLU_BWD) {
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const float sg = sigmoid_f(in[2 * j + 1]), x = in[2 * j];
      out[2 * j] = v[j] * sg;
      out[2 * j + 1] = v[j] * x * sg * (1.0f - sg);
    }
  }
}

// (x, y) times (the floats with bits fx, fy), then both times s: two packed products. Taking a scale per column apart costs the
// epilogue as many instructions as the packed form saves it.
__device__ __forceinline__ void scale_pair(float& x, float& y, uint32_t fx, uint32_t fy, float s) {
  asm("{ .reg .b64 v, f, t;\n\t"
      "mov.b64 v, {%0, %1};\n\tmov.b64 f, {%2, %3};\n\tmov.b64 t, {%4, %4};\n\t"
      "mul.rn.f32x2 v, v, f;\n\tmul.rn.f32x2 v, v, t;\n\tmov.b64 {%0, %1}, v; }"
      : "+f"(x), "+f"(y) : "r"(fx), "r"(fy), "f"(s));
}

// A thread's row of a chunk to and from its tile in shared memory.
template <int n>
__device__ __forceinline__ void chunk_put(uint8_t* tile, int r, const float* x) {
#pragma unroll
  for (int j = 0; j < n; j += 4)
    *reinterpret_cast<float4*>(tile + swizzled<4 * n>(r, j / 4)) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
}
template <int n>
__device__ __forceinline__ void chunk_get(const uint8_t* tile, int r, float* x) {
#pragma unroll
  for (int j = 0; j < n; j += 4) {
    const float4 q = *reinterpret_cast<const float4*>(tile + swizzled<4 * n>(r, j / 4));
    x[j] = q.x, x[j + 1] = q.y, x[j + 2] = q.z, x[j + 3] = q.w;
  }
}

// One GEMM of a launch: its arguments, what undoes the scales of the weight's rows, its tensor maps.
struct Side {
  CUtensorMap map_a, map_b, map_blo, map_in, map_c, map_pre;
  GemmArgs p;
  const uint16_t* b_unscale;
};
// SIDES = 2: two GEMMs of one epilogue that do not depend on each other, the atoms' and the edges' of a step of the network. The
// atoms' have few tiles, each with the longer contraction, and alone leave most SMs idle. Side 0's tiles go first. `rounds` is how
// many of side 1's tiles take about as long as one of side 0's: the workers that have no tile in side 0's last, partial round take
// that many of side 1's in the meantime. Measured, one after the other -> together: 1728 atoms, FMT_F16X2, SwiGLU 246 us -> 219,
// w_out 138 -> 107, heads 92 -> 77, backward of w_in 214 -> 167; a pass of 21 atoms 1069 us -> 928, of 648 (native) 4.84 ms -> 4.67.
struct Walk {
  int workers, n0, n1, full, lead, others, rounds;  // n0, n1 the sides' tiles, full and lead side 0's whole rounds and the rest
  __host__ __device__ Walk() {}
  __host__ Walk(int workers, int n0, int n1, int rounds)
      : workers(workers), n0(n0), n1(n1), full(n0 / workers), lead(n0 % workers), others(lead ? workers - lead : 0), rounds(rounds) {}
  // Worker w's k-th tile (once false, false for every later k).
  __host__ __device__ bool at(int w, int k, int& side, int& t) const {
    const bool between = lead > 0 && w >= lead;
    const int j = k - full - (w < lead ? 1 : 0);
    side = j < 0 ? 0 : 1;
    if (j < 0) t = w + k * workers;
    else if (between && j < rounds) t = w - lead + j * others;
    else t = rounds * others + w + (j - (between ? rounds : 0)) * workers;
    return t < (j < 0 ? n0 : n1);
  }
};
template <int SIDES>
struct Sides {
  Side side[SIDES];
  Walk walk;
};

template <int EPI, int BN, int FMT, bool PAIR, bool SPLIT, int SIDES>
__global__ void __launch_bounds__(Tile<BN, FMT, PAIR>::kThreads, 1) k_gemm_tc(const __grid_constant__ Sides<SIDES> g, int* err) {
  using L = Tile<BN, FMT, PAIR>;
  constexpr int NA = L::NA, NB = L::NB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring_a = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* ring_b = ring_a + NA * L::kA;
  uint8_t* epi = ring_a + L::kRings;
  // Barriers of a step, in a ring as long as A's (B's is no longer, so a barrier's phase is over before B's next use of it).
  // In a pair, `ready` and `tempty` are the leader's (rank 0), whose warp 1 issues the products of both; the commits of
  // those arrive in both CTAs.
  uint64_t* full_a = reinterpret_cast<uint64_t*>(epi + L::kEpi);  // [NA] the fp32 slab has landed (pair: and B's tile)
  uint64_t* ready = full_a + NA;    // [NS] it has been split and B's tile has landed (FMT_TF32: both have landed)
  uint64_t* done = ready + L::NS;   // [ND] the step's products are done
  uint64_t* empty_a = done + L::ND;                // TA: [NA] the slab has been read
  uint64_t* tfull = empty_a + (L::TA ? NA : 0);    // [2] accumulator complete
  uint64_t* tempty = tfull + 2;     // [2] accumulator read back
  uint64_t* landed = tempty + 2;    // [kEpiWarps][2] an epilogue warp's chunk has landed
  uint64_t* squares_there = landed + 2 * kEpiWarps;  // RMSNorm: a tile's rows' sums of squares are there,
  uint64_t* squares_read = squares_there + 1;        // and have been read
  float* squares = reinterpret_cast<float*>(epi + L::kEpi + L::kBars);  // [2][TBM]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(squares_read + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // A pair walks tiles of 2 x 128 rows: its CTAs take 128 each, and half of B's rows each.
  constexpr int CTAS = PAIR ? 2 : 1;
  const int rank = PAIR ? int(cluster_ctarank()) : 0;
  const auto tiles_n = [&](const GemmArgs& p) { return (p.N + BN - 1) / BN; };
  // SPLIT: the CTAs of a cluster share a tile; each sums a run of K, then finishes a slice of the columns. With two sides the
  // clusters past side 0's tiles take one of side 1's a CTA (or, past those, rows past the matrix).
  const int width = SPLIT ? int(cluster_size()) : 1, n0 = g.walk.n0;
  const bool shared = SPLIT && (SIDES == 1 || int(blockIdx.x) < n0 * width);
  const int me = SPLIT ? int(cluster_ctarank()) : 0, part = shared ? me : 0, parts = shared ? width : 1, slice = BN / parts;
  // This CTA's k-th tile: its side, the first row of this CTA's part of it, its first column.
  struct At {
    int side, row, col;
  };
  const auto at = [&](int k, At& x) {
    int t;
    bool have;
    if (SPLIT) {
      x.side = shared ? 0 : SIDES - 1, t = shared ? int(blockIdx.x) / width : int(blockIdx.x) - n0 * width;
      have = k == 0;
    } else if (SIDES == 1) {
      x.side = 0, t = int(blockIdx.x) / CTAS + k * g.walk.workers;
      have = t < g.walk.n0;
    } else {
      // Asked for anew each time: what follows from it, kept over a role's loop, has FMT_F16X3's sums spilled (600 bytes a thread).
      int w;
      asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(w));
      have = g.walk.at(w / CTAS, k, x.side, t);
    }
    const int tn = tiles_n(g.side[x.side].p);
    x.row = (t / tn * CTAS + rank) * TBM, x.col = t % tn * BN;
    return have;
  };
  constexpr int TBK = L::BK;
  // RMSNorm before the product (GemmArgs::rms). The converter, which sees every value of a row, adds up its squares; the epilogue
  // scales. 122138 rows, FMT_F16X2, norm and attention's input layer 169 us -> 143; the edges' SwiGLU 254 -> 260 with the atoms' tiles in
  // it; and a launch of 4 us less on a small structure's chain. (Sums of squares left in memory by the GEMM before cost it 10-18 us
  // and this one, which has to wait for them, 35-45.) A step's squares are summed by themselves: in one chain over K the sum's error
  // grew with K (1 / rms of 1024 normal values 1.17 of 2^-24 off, root mean square over the rows, and of 256 0.85; now 0.65 and
  // 0.58, a warp's norm by itself 0.75 and 0.73).
  constexpr bool kNorms = (EPI == EPI_PLAIN || EPI == EPI_SWIGLU) && !SPLIT && (L::X3 || L::X2 || L::T2);
  static_assert(!kNorms || L::kGroups == 2, "two sums a row");
  // SPLIT: parts divides the steps of K
  const auto steps = [&](const GemmArgs& p) { return (p.K + TBK - 1) / TBK / parts; };

  // The maps on their way while the kernel before this one still runs: the first load through one waits for it.
  if (warp == 3)
    for (int i = lane; i < 6 * SIDES; i += 32) prefetch_map(&g.side[i / 6].map_a + i % 6);
  if (threadIdx.x == 0) {
    for (int s = 0; s < NA; ++s) mbar_init(full_a + s, CTAS);
    if (L::TA)
      for (int s = 0; s < NA; ++s) mbar_init(empty_a + s, 4);
    for (int s = 0; s < L::NS; ++s)
      mbar_init(ready + s, L::TA ? 1 + 4 : PAIR ? 2 * (4 / L::kGroups) : 1 + (L::T1 ? 1 : 4 / L::kGroups));
    for (int s = 0; s < L::ND; ++s) mbar_init(done + s, 1);
    for (int b = 0; b < 2; ++b) mbar_init(tfull + b, 1), mbar_init(tempty + b, CTAS * kEpiWarps);
    for (int b = 0; b < 2 * kEpiWarps; ++b) mbar_init(landed + b, 1);
    mbar_init(squares_there, L::TA ? 8 : 4), mbar_init(squares_read, kEpiWarps);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc<PAIR>(tmem_slot, L::kColumns);  // accumulators of BN fp32 columns x 128 lanes
  tcgen05_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // the other CTA's barriers exist before anything signals them
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_slot;
  after_previous();

  // A converter lane's squares of a step's columns of a row, four at a time; and the sums of a tile's rows handed over to the
  // epilogue, by a warp for `n` rows a lane, `step` apart.
  const auto add_squares = [](float* sq, const float4& v) {
    asm("{ .reg .b64 s, a, b;\n\tmov.b64 s, {%0, %1};\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "fma.rn.f32x2 s, a, a, s;\n\tfma.rn.f32x2 s, b, b, s;\n\tmov.b64 {%0, %1}, s; }"
        : "+f"(sq[0]), "+f"(sq[1]) : "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
  };
  const auto hand_over = [&](int norms, int group, int r, int step, const float (*sq)[2], int n) {
    if (norms > 0 && !mbar_wait_warp(squares_read, (norms - 1) & 1, abort_flag)) return false;
    for (int j = 0; j < n; ++j) squares[group * TBM + r + j * step] = sq[j][0] + sq[j][1];
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(squares_there);
    return true;
  };

  if (warp < 4) {
    if (L::kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(L::kRegsProd));
    // Each of the three roles is a whole warp's loop with one lane's instructions. `s` is the step's slot in its ring, `turn`
    // the parity of the ring's round.
    const bool one = elect_one();
    bool ok = true;
    if (warp == 0) {
      uint64_t* freed = L::TA ? empty_a : done;
      int s = 0;
      uint32_t turn = 0;
      bool peek = true;
      At x;
      for (int k = 0; ok && at(k, x); ++k) {
        const Side& q = g.side[x.side];
        const int kb0 = part * steps(q.p), kb1 = kb0 + steps(q.p);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!(ok = mbar_wait_warp(freed + s, turn ^ 1, abort_flag, peek))) break;
          peek = s + 1 < NA ? mbar_test(freed + s + 1, turn ^ 1) : mbar_test(freed, turn);
          if (one) {
            uint64_t* bar = L::T1 ? ready + s : full_a + s;
            mbar_expect_tx(bar, uint32_t(box_rows(q.p.M) * L::BK * 4));
            tma_load_2d(ring_a + s * L::kA, &q.map_a, bar, kb * TBK, x.row);
          }
          if (++s == NA) s = 0, turn ^= 1;
        }
      }
    } else if (warp == 2) {
      int s = 0, sb = 0, gone = 0;  // the step's barrier, B's slot, steps so far
      bool peek = false;
      At x;
      for (int k = 0; ok && at(k, x); ++k) {
        const Side& q = g.side[x.side];
        const int first = x.col + rank * L::kRowsB, kb0 = part * steps(q.p), kb1 = kb0 + steps(q.p);
        for (int kb = kb0; kb < kb1; ++kb, ++gone) {
          // the step that used this slot before, NB steps ago, has its barrier at (gone - NB) % ND
          if (gone >= NB && !(ok = mbar_wait_warp(done + (gone - NB) % L::ND, ((gone - NB) / L::ND) & 1, abort_flag, peek))) break;
          if (gone + 1 >= NB) peek = mbar_test(done + (gone + 1 - NB) % L::ND, ((gone + 1 - NB) / L::ND) & 1);
          if (one) {
            uint8_t* dst = ring_b + sb * L::kB;
            uint64_t* bar = PAIR ? full_a + s : ready + s;
            mbar_expect_tx(bar, L::kB);
            if (L::X3 || L::X2) {
              tma_load_2d(dst, &q.map_b, bar, kb * 64, first);
              if (L::X3) tma_load_2d(dst + L::kRowsB * 128, &q.map_blo, bar, kb * TBK, first);
            } else {
              tma_load_2d(dst, &q.map_b, bar, kb * TBK, first);
              if (L::T2) tma_load_2d(dst + L::kRowsB * 64, &q.map_blo, bar, kb * TBK, first);
            }
          }
          if (++s == L::NS) s = 0;
          if (++sb == NB) sb = 0;
        }
      }
    } else if (warp == 1 && rank == 0) {
      constexpr uint32_t idesc = L::T2 || L::T1 ? idesc_tf32(CTAS * TBM, BN) : idesc_f16(CTAS * TBM, BN, FMT == FMT_BF16);
      int s = 0, sb = 0, sd = 0, i = 0, run = 0;  // the slots, accumulators handed over, steps into this one
      uint32_t turn = 0;
      bool peek = false;
      At x;
      for (int k = 0; ok && at(k, x); ++k) {
        const GemmArgs& p = g.side[x.side].p;
        const int kb0 = part * steps(p), kb1 = kb0 + steps(p), drain = L::drain(p.K);
        for (int kb = kb0; kb < kb1; ++kb) {
          const bool first = run == 0, last = kb + 1 == kb1 || run + 1 == drain;
          const int b = i % L::kTurns;
          if (first) {
            if (!(ok = mbar_wait_warp(tempty + b, ((i / L::kTurns) & 1) ^ 1, abort_flag))) break;
            tcgen05_fence_after();
          }
          if (!(ok = mbar_wait_warp(ready + s, turn, abort_flag, peek))) break;
          peek = s + 1 < L::NS ? mbar_test(ready + s + 1, turn) : mbar_test(ready, turn ^ 1);
          if (L::TA) tcgen05_fence_after();
          if (L::TA && one) {
            const uint32_t acc = tmem + uint32_t(b * L::kAccs * BN), b0 = smem_u32(ring_b + sb * L::kB);
            const uint32_t th = tmem + uint32_t(L::kPartsAt + s * 16 * L::kParts);
            constexpr int row = L::X3 || L::X2 ? 128 : 64;
            const uint64_t bh = smem_desc<row>(b0), bm = smem_desc<row>(b0 + 64);
#pragma unroll
            for (int k = 0; k < 4; k += 2) {  // 16 columns: 8 of tensor memory, and as below
              const uint32_t h = th + 4 * k, m = h + 16, l = h + 32;
              if (L::X3) {
                const uint64_t bl = smem_desc<64>(b0 + L::kRowsB * 128);
                const uint32_t small = acc + BN;
                if (L::kFull) mma_f16_ta(small, m, bl + k, idesc, !first || k != 0), mma_f16_ta(small, l, bm + k, idesc, 1);
                mma_f16_ta(small, h, bl + k, idesc, L::kFull || !first || k != 0);
                mma_f16_ta(small, l, bh + k, idesc, 1);
                mma_f16_ta(small, m, bm + k, idesc, 1);
                mma_f16_ta(small, h, bm + k, idesc, 1);
                mma_f16_ta(small, m, bh + k, idesc, 1);
                mma_f16_ta(acc, h, bh + k, idesc, !first || k != 0);
              } else if (L::X2) {
                mma_f16_ta(acc, h, bm + k, idesc, kb != kb0 || k != 0);
                mma_f16_ta(acc, m, bh + k, idesc, 1);
                mma_f16_ta(acc, h, bh + k, idesc, 1);
              } else {
                mma_f16_ta(acc, h, bh + k, idesc, kb != kb0 || k != 0);
              }
            }
            mma_commit<false>(done + sd);
            if (last) mma_commit<false>(tfull + b);
          }
          if (!L::TA && one) {
            const uint32_t acc = tmem + uint32_t(b * L::kAccs * BN);
            const uint32_t a0 = smem_u32(ring_a + s * L::kA), b0 = smem_u32(ring_b + sb * L::kB);
            const uint64_t ah = smem_desc<128>(a0), am = smem_desc<128>(a0 + 64);  // h and the part beside it
            if (L::X3) {
              const uint64_t al = smem_desc<64>(a0 + TBM * 128), bh = smem_desc<128>(b0), bm = smem_desc<128>(b0 + 64),
                             bl = smem_desc<64>(b0 + L::kRowsB * 128);
              const uint32_t small = acc + BN;
#pragma unroll
              for (int k = 0; k < 4; k += 2) {  // 16 columns are 32 bytes: 2 in the descriptors' 16-byte units
                if (L::kFull) mma_f16<PAIR>(small, am + k, bl + k, idesc, !first || k != 0), mma_f16<PAIR>(small, al + k, bm + k, idesc, 1);
                mma_f16<PAIR>(small, ah + k, bl + k, idesc, L::kFull || !first || k != 0);
                mma_f16<PAIR>(small, al + k, bh + k, idesc, 1);
                mma_f16<PAIR>(small, am + k, bm + k, idesc, 1);
                mma_f16<PAIR>(small, ah + k, bm + k, idesc, 1);
                mma_f16<PAIR>(small, am + k, bh + k, idesc, 1);
                mma_f16<PAIR>(acc, ah + k, bh + k, idesc, !first || k != 0);
              }
            } else if (L::X2) {
              const uint64_t bh = smem_desc<128>(b0), bl = smem_desc<128>(b0 + 64);
#pragma unroll
              for (int k = 0; k < 4; k += 2) {
                mma_f16<PAIR>(acc, ah + k, bl + k, idesc, kb != kb0 || k != 0);
                mma_f16<PAIR>(acc, am + k, bh + k, idesc, 1);
                mma_f16<PAIR>(acc, ah + k, bh + k, idesc, 1);
              }
            } else if (L::T2) {
              const uint64_t th = smem_desc<64>(a0), tl = smem_desc<64>(a0 + L::kSlab), bh = smem_desc<64>(b0), bl = smem_desc<64>(b0 + L::kRowsB * 64);
#pragma unroll
              for (int k = 0; k < 4; k += 2) {  // 8 columns are 32 bytes
                mma_tf32<PAIR>(acc, th + k, bl + k, idesc, kb != kb0 || k != 0);
                mma_tf32<PAIR>(acc, tl + k, bh + k, idesc, 1);
                mma_tf32<PAIR>(acc, th + k, bh + k, idesc, 1);
              }
            } else if (L::T1) {
              const uint64_t bh = smem_desc<128>(b0);
#pragma unroll
              for (int k = 0; k < 8; k += 2) mma_tf32<PAIR>(acc, ah + k, bh + k, idesc, kb != kb0 || k != 0);
            } else {
              const uint64_t bh = smem_desc<64>(b0);
#pragma unroll
              for (int k = 0; k < 4; k += 2) mma_f16<PAIR>(acc, ah + k, bh + k, idesc, kb != kb0 || k != 0);
            }
            mma_commit<PAIR>(done + s);
            if (last) mma_commit<PAIR>(tfull + b);
          }
          __syncwarp();
          i += last, run = last ? 0 : run + 1;
          if (++s == L::NS) s = 0, turn ^= 1;
          if (++sb == NB) sb = 0;
          if (++sd == L::ND) sd = 0;
        }
      }
    }
  } else if (warp < kConvWarp0) {
    if (L::kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(L::kRegsEpi));
    const int ew = warp - kEpiWarp0;
    const int q = warp & 3;          // the quarter of the 128 lanes this warp may read
    const int half = ew >> 2;        // which half of the BN columns
    constexpr int W = L::kWide, AC = EPI == EPI_SWIGLU_BWD ? W / 2 : W;  // columns of a buffer, of accumulator a chunk takes
    constexpr int CW = EPI == EPI_SWIGLU ? W / 2 : W;                    // columns of C a chunk gives
    uint8_t* buf = epi + ew * 2 * L::kBuf;
    uint64_t* bar = landed + 2 * ew;
    const bool has_in = reads(EPI) && (EPI != EPI_PLAIN || g.side[0].p.res != nullptr);  // (both sides read, or neither)
    // The chunks of a warp: its half of the columns; SPLIT: every other one of the CTA's slice.
    auto first_col = [&](const At& x) { return x.col + (SPLIT ? part * slice : half * (BN / 2)); };
    auto chunks_of = [&](const At& x) { return max(0, min((SPLIT ? slice : BN / 2) / AC, (g.side[x.side].p.N - first_col(x) + AC - 1) / AC)); };
    const int c0 = SPLIT ? half : 0;
    constexpr int CS = SPLIT ? 2 : 1;
    auto ask = [&](const At& x, int c, int k) {  // lane 0: chunk c of tile x, the k-th this warp reads, into buffer k & 1
      mbar_expect_tx(bar + (k & 1), L::kBuf);
      tma_load_2d(buf + (k & 1) * L::kBuf, &g.side[x.side].map_in, bar + (k & 1), (first_col(x) + c * AC) * (W / AC), x.row + q * 32);
    };
    auto ask_first = [&](int from, int k) {  // the same for the first chunk of the first tile from this CTA's from-th on that has one
      At y;
      for (; at(from, y); ++from)
        if (chunks_of(y) > c0) return ask(y, c0, k);
    };
    auto release = [&](int b) {  // the accumulators of turn b have been read: the issuer may reuse them
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_at(tempty + b, 0);
        else mbar_arrive(tempty + b);
      }
    };
    int i = 0, k = 0, norms = 0;  // accumulators, chunks and tiles after a norm so far
    const auto row_max = [&](int tile) {  // of this thread's row of a tile
      At y;
      if (!L::kScaled || !at(tile, y)) return 0u;
      const GemmArgs& p = g.side[y.side].p;
      return __ldg(p.a_max + min(y.row + q * 32 + lane, p.M - 1));
    };
    // asked for a tile ahead (FMT_F16X3, which has no register to spare, waits longer for its sums than for this)
    uint32_t next_max = L::X3 ? 0 : row_max(0);
    bool ok = true;
    if (has_in && lane == 0) ask_first(0, 0);
    const auto finish = [&](const Side& sd, int tile, const At& x) {
      const GemmArgs& p = sd.p;
      const int r0 = x.row + q * 32, row = r0 + lane, n0 = first_col(x), nc = chunks_of(x);
      if (reads(EPI)) epilogue_prefetch<EPI>(p, row, n0, BN / 2);
      // The scales of a chunk's columns. FMT_F16X3, whose epilogue threads have registers to spare (and whose launches are the
      // small structures'), asks for them a chunk ahead, the first ones while the accumulator is being filled: asked for where
      // they are used they cost each launch of a 21-atom pass 0.7 us. The others, whose chunks are twice as wide, would spill.
      // A scale per row against one for the matrix: GEMMs of diamond1728 3xTF32 7.57 -> 7.63 ms, of water1791 tf32 4.12 -> 4.19,
      // of water648 native 3.86 -> 3.90.
      constexpr bool kAhead = L::X3;
      uint4 u[L::kScaled ? AC / 8 : 1];
      const auto ask_scales = [&](int c) {
        if (L::kScaled)
#pragma unroll
          for (int j = 0; j < AC / 8; ++j)
            if (c < nc && n0 + c * AC + 8 * j < p.N) u[j] = __ldg(reinterpret_cast<const uint4*>(sd.b_unscale + n0 + c * AC + 8 * j));
      };
      if (kAhead) ask_scales(c0);
      float big = 0.f;
      RowTerms rt{};
      if (row < p.M) {
        if (EPI == EPI_COMPRESS) {
          rt.tab = p.tab + size_t(p.sp[row]) * p.N;
          rt.e0 = (float) p.vec[3 * size_t(row)], rt.e1 = (float) p.vec[3 * size_t(row) + 1], rt.e2 = (float) p.vec[3 * size_t(row) + 2];
          rt.e3 = (float) p.dist[row];
        }
      } else if (EPI == EPI_COMPRESS) {
        rt.tab = p.tab;
      }
      float unscale = 1.f;
      if (L::X3) {
        if (row < p.M) unscale = unscale_of(p.a_max[row]);
      } else {
        if (L::kScaled) unscale = unscale_of(next_max);
        next_max = row_max(tile + 1);
      }
      float sum[L::kSums];
      uint32_t acc = 0;
      const auto accumulator = [&](int b) { return tmem + uint32_t(b * L::kAccs * BN + half * (BN / 2)) + (uint32_t(q * 32) << 16); };
      if (L::X3 && !SPLIT) {
        // a piece of K at a time (drain); the first by itself: as a pass of the loop it has the sums spilled where K is per side
        const auto piece = [&](auto add) {
          const int b = i % L::kTurns;
          if (!(ok = mbar_wait_warp(tfull + b, (i / L::kTurns) & 1, abort_flag))) return;
          tcgen05_fence_after();
          acc = accumulator(b);
#pragma unroll
          for (int c = 0; c < L::kSums; c += 16) {
            uint32_t big16[16], small16[16];
            tmem_ld16_async(acc + c, big16);
            tmem_ld16_async(acc + BN + c, small16);
            tmem_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float v = __uint_as_float(big16[j]) + __uint_as_float(small16[j]);
              sum[(c + j) % L::kSums] = add ? sum[(c + j) % L::kSums] + v : v;
            }
          }
          release(b);
          ++i;
        };
        piece(std::false_type());
#pragma unroll 1
        for (int kb = L::drain(p.K); ok && kb < steps(p); kb += L::drain(p.K)) piece(std::true_type());
        if (!ok) return;
      } else {
        const int b = i % L::kTurns;
        ok = mbar_wait_warp(tfull + b, (i / L::kTurns) & 1, abort_flag);
        if (!ok && !SPLIT) return;
        tcgen05_fence_after();
        acc = accumulator(b);
      }
      // SPLIT: where the rings were, each CTA gets its slice of every CTA's sums, four columns of 32 rows at a time. (One tile a
      // CTA: nothing else is under way then, and the two barriers are met by every thread whatever happened.)
      const auto piece = [&](int from, int run) {
        return reinterpret_cast<float4*>(ring_a) + (size_t(from * 4 + q) * (slice / 4) + run) * 32 + lane;
      };
      if constexpr (SPLIT) {
        cluster_sync_all();
        if (ok) {
#pragma unroll
          for (int c = 0; c < BN / 2; c += 16) {
            float y[16];
            tmem_ld<16>(acc + c, y);
            if (L::X3) {  // (one piece a CTA)
              float small[16];
              tmem_ld<16>(acc + BN + c, small);
#pragma unroll
              for (int j = 0; j < 16; ++j) y[j] += small[j];
            }
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const int col = half * (BN / 2) + c + j;
              store4_at(piece(part, col % slice / 4), shared ? col / slice : me, y[j], y[j + 1], y[j + 2], y[j + 3]);
            }
          }
        }
        cluster_sync_all();
        if (!ok) return;
      }
      if (kNorms && p.rms != 0.f) {
        if (!(ok = mbar_wait_warp(squares_there, norms & 1, abort_flag))) return;
        // (a row's largest value over its root mean square lies in [1, sqrt K]: the product with its scale is a normal number)
        unscale *= reciprocal_root(fmaf(squares[q * 32 + lane] + squares[TBM + q * 32 + lane], p.rms, kRmsEps));
        __syncwarp();
        if (lane == 0) mbar_arrive(squares_read);
        ++norms;
      }
      // One copy of the chunk's code; FMT_F16X3 moves its sums down after each chunk: unrolled, the compiler keeps every
      // chunk's addresses alive beside the sums and spills.
#pragma unroll 1
      for (int c = c0; c < nc; c += CS) {
        float v[AC], in[W], out[W], pre[W];
        if (!kAhead) ask_scales(c);
        if constexpr (SPLIT) {
#pragma unroll
          for (int j = 0; j < AC; j += 4) {
            float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int o = 0; o < parts; ++o) {  // in K's order
              const float4 y = *piece(o, (c * AC + j) / 4);
              z = o == 0 ? y : make_float4(z.x + y.x, z.y + y.y, z.z + y.z, z.w + y.w);
            }
            v[j] = z.x, v[j + 1] = z.y, v[j + 2] = z.z, v[j + 3] = z.w;
          }
        } else if (L::X3) {
#pragma unroll
          for (int j = 0; j < AC; ++j) v[j] = sum[j % L::kSums];
#pragma unroll
          for (int j = 0; j + AC < L::kSums; ++j) sum[j] = sum[j + AC];
        } else {
          tmem_ld<AC == 32 ? 32 : 16>(acc + c * AC, v);
          if (c + 1 == nc) release(i % L::kTurns);  // (not SPLIT)
        }
        if (L::kScaled) {
#pragma unroll
          for (int j = 0; j < AC; j += 8) {
            const uint32_t two[4] = {u[j / 8].x, u[j / 8].y, u[j / 8].z, u[j / 8].w};
#pragma unroll
            for (int i = 0; i < 4; ++i)  // one after the other: the two scales' product may not be a normal number
              scale_pair(v[j + 2 * i], v[j + 2 * i + 1], two[i] << 16, two[i] & 0xFFFF0000u, unscale);
          }
          if (kAhead) ask_scales(c + CS);
        } else if (kNorms && p.rms != 0.f) {
#pragma unroll
          for (int j = 0; j < AC; ++j) v[j] *= unscale;
        }
        uint8_t* mine = buf + (k & 1) * L::kBuf;
        if (has_in) {
          if (lane == 0) {
            bulk_wait_read<0>();  // the chunk before this one has left the other buffer: the next one may come in
            if (c + CS < nc) ask(x, c + CS, k + 1);
            else ask_first(tile + 1, k + 1);
          }
          __syncwarp();
          if (!(ok = mbar_wait_warp(bar + (k & 1), (k >> 1) & 1, abort_flag))) return;
          chunk_get<W>(mine, lane, in);
        }
        epilogue_row<EPI, AC>(p, row, n0 + c * AC, rt, v, has_in, in, out, pre);
#pragma unroll
        for (int j = 0; j < CW; ++j) big = fmaxf(big, fabsf(out[j]));
        if (!has_in) {
          if (lane == 0) {
            if (writes_two(EPI)) bulk_wait_read<0>();
            else bulk_wait_read<1>();
          }
          __syncwarp();
        }
        if (writes_two(EPI)) {
          if (p.pre) chunk_put<W>(buf, lane, pre);
          mine = buf + L::kBuf;
        }
        if (EPI != EPI_SWIGLU || p.C) chunk_put<CW>(mine, lane, out);
        fence_async_smem();
        __syncwarp();
        if (lane == 0 && r0 < p.M) {
          if (writes_two(EPI) && p.pre) tma_store_2d(&sd.map_pre, buf, n0 + c * AC, r0);
          if (EPI != EPI_SWIGLU || p.C) tma_store_2d(&sd.map_c, mine, (n0 + c * AC) * CW / AC, r0);
          bulk_commit();
        }
        ++k;
      }
      if (!L::X3) {
        if (!SPLIT && nc == 0) release(i % L::kTurns);
        ++i;
      }
      if (p.c_max && row < p.M && nc > 0) atomicMax(p.c_max + row, __float_as_uint(big));
    };
    At x;
    for (int tile = 0; ok && at(tile, x); ++tile) {
      finish(g.side[SIDES == 1 ? 0 : x.side], tile, x);
    }
    if (lane == 0) bulk_wait_all();
  } else if (L::TA) {
    if (L::kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(L::kRegsConv));
    // A lane owns one of its warp's quarter of the rows; the groups take every other step.
    const int quarter = warp & 3, group = (warp - kConvWarp0) >> 2;
    int gone = 0, norms = 0;
    bool ok = true, peek = false;
    const int r = quarter * 32 + lane;
    const auto row_max = [&](int k) {
      At y;
      if (!L::kScaled || !at(k, y)) return 0u;
      const GemmArgs& p = g.side[y.side].p;
      return y.row + r < p.M ? __ldg(p.a_max + y.row + r) : 0u;
    };
    uint32_t next = row_max(0);  // asked for a tile ahead: HBM is a sixth of a tile's time away
    At x;
    for (int k = 0; ok && at(k, x); ++k) {
      const GemmArgs& p = g.side[x.side].p;
      const int row = x.row + r, kb0 = part * steps(p), kb1 = kb0 + steps(p);
      const bool live = row - lane < p.M;  // rows past the matrix: whatever their products are, nobody reads them
      const float s = L::kScaled ? scale_of(next) : 1.f;
      next = row_max(k + 1);
      float sq[1][2] = {{0.f, 0.f}};
      for (int kb = kb0; kb < kb1; ++kb, ++gone) {
        if ((gone & 1) != group) continue;
        const int sa = gone % NA, sp = gone % L::NS, before = gone - L::NS;
        if (!(ok = mbar_wait_warp(full_a + sa, (gone / NA) & 1, abort_flag, peek))) break;
        const bool free_peek = before < 0 || mbar_test(done + before % L::ND, (before / L::ND) & 1);
        peek = mbar_test(full_a + (gone + 2) % NA, ((gone + 2) / NA) & 1);
        uint32_t part[3][16];
        float of_step[2] = {0.f, 0.f};
        if (live) {
          const uint8_t* slab = ring_a + sa * L::kA;
          float4 v[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) v[c] = *reinterpret_cast<const float4*>(slab + swizzled<128>(r, c));
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            if (kNorms && p.rms != 0.f) add_squares(of_step, v[c]);
            split2<FMT>(v[c].x, v[c].y, s, part[0][2 * c], part[1][2 * c], part[2][2 * c]);
            split2<FMT>(v[c].z, v[c].w, s, part[0][2 * c + 1], part[1][2 * c + 1], part[2][2 * c + 1]);
          }
          if (kNorms) sq[0][0] += of_step[0], sq[0][1] += of_step[1];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_a + sa);
        if (!(ok = mbar_wait_warp(done + before % L::ND, (before / L::ND) & 1, abort_flag, free_peek))) break;
        tcgen05_fence_after();
        if (live) {
          const uint32_t at = tmem + uint32_t(L::kPartsAt + sp * 16 * L::kParts) + (uint32_t(quarter * 32) << 16);
#pragma unroll
          for (int q = 0; q < L::kParts; ++q) tmem_st16_async(at + 16 * q, part[q]);
          tmem_wait_st();
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ready + sp);
      }
      if (ok && kNorms && p.rms != 0.f) ok = hand_over(norms++, group, r, 0, sq, 1);
    }
  } else if (!L::T1) {
    if (L::kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(L::kRegsConv));
    // A lane owns a row at a time: 16-byte chunk c of row r sits at chunk c ^ (r & 7) of its 128 bytes, so the eight lanes of
    // a quarter warp touch eight different 16-byte columns on the reads and on the writes. The parts go back as chunks 0-3
    // (h) and 4-7 (m or l) of the same row; FMT_F16X3's l into rows of 64 bytes, chunk c at c ^ ((r >> 1) & 3).
    constexpr int WPG = 4 / L::kGroups;  // warps of a group
    const int cw = warp - kConvWarp0, group = cw / WPG, first = cw % WPG;
    int gone = 0, norms = 0;
    bool ok = true, peek = false;
    uint32_t next[4 / WPG];  // the rows' maxima, asked for a tile ahead
    const auto row_max = [&](int k) {
      At y;
      const bool have = L::kScaled && at(k, y);
#pragma unroll
      for (int j = 0; j < 4 / WPG; ++j) {
        const int row = have ? y.row + (first + j * WPG) * 32 + lane : 0;
        next[j] = have && row < g.side[y.side].p.M ? __ldg(g.side[y.side].p.a_max + row) : 0;
      }
    };
    row_max(0);
    At x;
    for (int k = 0; ok && at(k, x); ++k) {
      const GemmArgs& p = g.side[x.side].p;
      const int m0 = x.row, kb0 = part * steps(p), kb1 = kb0 + steps(p);
      float scale[4 / WPG];
#pragma unroll
      for (int j = 0; j < 4 / WPG; ++j) scale[j] = L::kScaled ? scale_of(next[j]) : 1.f;
      row_max(k + 1);
      float sq[4 / WPG][2] = {};
      for (int kb = kb0; kb < kb1; ++kb, ++gone) {
        if (gone % L::kGroups != group) continue;
        const int sa = gone % NA;
        if (!(ok = mbar_wait_warp(full_a + sa, (gone / NA) & 1, abort_flag, peek))) break;
        peek = mbar_test(full_a + (gone + L::kGroups) % NA, ((gone + L::kGroups) / NA) & 1);
        uint8_t* slab = ring_a + sa * L::kA;
#pragma unroll
        for (int j = 0; j < 4 / WPG; ++j) {
          const int r = (first + j * WPG) * 32 + lane;
          if (m0 + r - lane >= p.M) break;  // rows past the matrix: whatever their products are, nobody reads them
          float of_step[2] = {0.f, 0.f};
          if (L::T2) {  // the slab is h; l goes beside it at the same place
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float4 v = *reinterpret_cast<const float4*>(slab + swizzled<64>(r, c));
              if (kNorms && p.rms != 0.f) add_squares(of_step, v);
              *reinterpret_cast<float4*>(slab + L::kSlab + swizzled<64>(r, c)) =
                  make_float4(tf32_low(v.x), tf32_low(v.y), tf32_low(v.z), tf32_low(v.w));
            }
            if (kNorms) sq[j][0] += of_step[0], sq[j][1] += of_step[1];
            continue;
          }
          const float s = scale[j];
          float4 v[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) v[c] = *reinterpret_cast<const float4*>(slab + swizzled<128>(r, c));
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 h, m, l;
            const float4 a = v[2 * c], b = v[2 * c + 1];
            if (kNorms && p.rms != 0.f) add_squares(of_step, a), add_squares(of_step, b);
            split2<FMT>(a.x, a.y, s, h.x, m.x, l.x), split2<FMT>(a.z, a.w, s, h.y, m.y, l.y);
            split2<FMT>(b.x, b.y, s, h.z, m.z, l.z), split2<FMT>(b.z, b.w, s, h.w, m.w, l.w);
            *reinterpret_cast<uint4*>(slab + swizzled<128>(r, c)) = h;
            if (L::X3 || L::X2) *reinterpret_cast<uint4*>(slab + swizzled<128>(r, 4 + c)) = m;
            if (L::X3) *reinterpret_cast<uint4*>(slab + L::kSlab + swizzled<64>(r, c)) = l;
          }
          if (kNorms) sq[j][0] += of_step[0], sq[j][1] += of_step[1];
        }
        fence_async_smem();  // generic-proxy writes visible to the tensor core
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_at(ready + sa, 0);
          else mbar_arrive(ready + sa);
        }
      }
      if (ok && kNorms && p.rms != 0.f) ok = hand_over(norms++, group, first * 32 + lane, 32 * WPG, sq, 4 / WPG);
    }
  }
  if (SPLIT && (warp < kEpiWarp0 || warp >= kConvWarp0)) {
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  tcgen05_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // nobody leaves while the other CTA may still signal it or read its tiles
  if (warp == 1) tmem_dealloc<PAIR>(tmem, L::kColumns);
  if (threadIdx.x == 0 && *abort_flag) atomicExch(err, 1);
}

// ---- host side ---------------------------------------------------------------------------

// A row-major matrix as a tensor map: `dims` innermost first, `pitch` the byte strides of the outer ones, zero fill outside.
CUtensorMap make_map(CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* pitch,
                     const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
  CUtensorMap m;
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = tensor_state().encode(&m, type, rank, const_cast<void*>(base), dims, pitch, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw Error(5, "gemm: cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return m;
}
CUtensorMap map_2d(CUtensorMapDataType type, const void* base, int cols, int rows, size_t pitch_bytes, int box_cols, int box_rows,
                   CUtensorMapSwizzle swizzle) {
  const cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rows)}, pitch[1] = {cuuint64_t(pitch_bytes)};
  const cuuint32_t box[2] = {cuuint32_t(box_cols), cuuint32_t(box_rows)};
  return make_map(type, 2, base, dims, pitch, box, swizzle);
}

// As many pairs as the device holds at once (a pair needs two SMs of one GPC: fewer than half the SMs may fit), or the last
// pairs of a persistent kernel would start when the first ones end. `table` is the kernel's own.
template <class K>
int resident_pairs(K kernel, cudaLaunchConfig_t cfg, PerDevice<int>& table) {
  int dev = 0;
  cudaGetDevice(&dev);
  return table.get(dev, [&](int& n) {
    cfg.gridDim = dim3(unsigned(tensor_state().sms / 2 * 2));
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) n = tensor_state().sms / 2;
    n = std::min(n, tensor_state().sms / 2);
  });
}

// Side k of a launch, with its tensor maps.
template <int EPI, class L>
Side make_side(const GemmTask& q) {
  const GemmArgs& a = q.a;
  const PackedB& w = q.w;
  Side s;
  s.p = a, s.b_unscale = w.unscale;
  if (a.rms != 0.f) s.p.rms = 1.0f / a.K;
  s.map_a = map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, a.A, a.K, a.M, size_t(a.lda) * 4, L::BK, box_rows(a.M),
                   L::T2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B);
  const auto half = w.fmt == FMT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  if (L::T1) {
    s.map_b = map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, w.main, w.Kp, a.N, size_t(w.Kp) * 4, L::BK, L::kRowsB, CU_TENSOR_MAP_SWIZZLE_128B);
  } else if (L::T2) {
    s.map_b = map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, w.main, w.Kp, a.N, size_t(w.Kp) * 4, L::BK, L::kRowsB, CU_TENSOR_MAP_SWIZZLE_64B);
    s.map_blo = map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, w.low, w.Kp, a.N, size_t(w.Kp) * 4, L::BK, L::kRowsB, CU_TENSOR_MAP_SWIZZLE_64B);
  } else if (L::X3 || L::X2) {
    s.map_b = map_2d(half, w.main, 2 * w.Kp, a.N, size_t(w.Kp) * 4, 64, L::kRowsB, CU_TENSOR_MAP_SWIZZLE_128B);
    if (L::X3) s.map_blo = map_2d(half, w.low, w.Kp, a.N, size_t(w.Kp) * 2, L::BK, L::kRowsB, CU_TENSOR_MAP_SWIZZLE_64B);
  } else {
    s.map_b = map_2d(half, w.main, w.Kp, a.N, size_t(w.Kp) * 2, L::BK, L::kRowsB, CU_TENSOR_MAP_SWIZZLE_64B);
  }
  if (!L::X3 && !L::T2) s.map_blo = s.map_b;
  // the epilogue's chunks: 32 rows x kWide columns of what it reads and writes (C half as wide after a SwiGLU)
  constexpr int W = L::kWide;
  auto chunk = [&](const float* base, int cols, int ld, int wide) {
    return map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, base, cols, a.M, size_t(ld) * 4, wide, 32,
                  wide == 32 ? CU_TENSOR_MAP_SWIZZLE_128B : wide == 16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
  };
  s.map_in = s.map_c = s.map_pre = s.map_a;
  const int c_cols = EPI == EPI_SWIGLU ? a.N / 2 : EPI == EPI_SWIGLU_BWD ? 2 * a.N : a.N;
  if (a.C) s.map_c = chunk(a.C, c_cols, a.ldc, EPI == EPI_SWIGLU ? W / 2 : W);
  if (EPI == EPI_PLAIN && a.res) s.map_in = chunk(a.res, a.N, a.ldr, W);
  if (EPI == EPI_SILU_BWD || EPI == EPI_SWIGLU_BWD) s.map_in = chunk(a.pre, c_cols, a.ldp, W);
  if (writes_two(EPI) && a.pre) s.map_pre = chunk(a.pre, a.N, a.ldp, W);
  return s;
}

// How a launch is cut: the tiles' width, pairs of CTAs, the CTAs that share a tile (of side 0), side 1's tiles to one of side 0's,
// and about how long it takes (clocks).
struct Plan {
  int bn = 0, parts = 1, rounds = 1;
  bool pair = false;
  long long clocks = 0;
};

template <int EPI, int BN, int FMT, bool PAIR, bool SPLIT, int SIDES>
void launch_tc(Stream& st, const GemmTask* q, const Plan& plan) {
  using L = Tile<BN, FMT, PAIR>;
  static_assert(L::kTotal <= 227 * 1024, "the tile pipeline does not fit shared memory");
  static SmemOptIn opted;
  static PerDevice<int> pairs;
  auto kernel = k_gemm_tc<EPI, BN, FMT, PAIR, SPLIT, SIDES>;
  opt_in_shared_memory(kernel, L::kTotal, opted);
  Sides<SIDES> g;
  long long tiles[2] = {0, 0};
  for (int i = 0; i < SIDES; ++i) {
    g.side[i] = make_side<EPI, L>(q[i]);
    tiles[i] = (long long) cdiv(q[i].a.M, PAIR ? 2 * TBM : TBM) * cdiv(q[i].a.N, BN);
  }
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2] = {};
  cfg.blockDim = dim3(L::kThreads), cfg.dynamicSmemBytes = L::kTotal, cfg.stream = st.s, cfg.attrs = attr;
  if (SPLIT) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = plan.parts, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(unsigned((tiles[0] + cdiv(tiles[1], plan.parts)) * plan.parts));
  } else if (PAIR) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(unsigned(2 * std::min<long long>(tiles[0] + tiles[1], resident_pairs(kernel, cfg, pairs))));
  } else {
    cfg.gridDim = dim3(unsigned(std::min<long long>(tiles[0] + tiles[1], tensor_state().sms)));
  }
  attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see launch()
  attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  g.walk = Walk(int(cfg.gridDim.x) / (PAIR ? 2 : 1), int(tiles[0]), int(tiles[1]), plan.rounds);
  PETB_CUDA(cudaLaunchKernelEx(&cfg, kernel, g, st.gave_up));
  PETB_LAUNCH_CHECK(st);
}

// Clocks a step of 32 columns takes on a tile 256, 128 or 64 wide, however few tiles there are (see the head of this file).
template <int FMT>
constexpr int step_clocks(int i) {
  constexpr bool X3 = three_parts(FMT), T2 = FMT == FMT_TF32X2, two = FMT == FMT_F16X2;
  constexpr int clocks[3] = {X3 || T2 ? 1800 : two ? 850 : 640, X3 ? 1050 : T2 ? 1550 : two ? 700 : 530, X3 ? 850 : T2 ? 1500 : two ? 670 : 510};
  return clocks[i];
}
// The same of a launch that fills the SMs, as measured: what two GEMMs in one launch are weighed by.
template <int FMT>
constexpr int full_clocks(int bn, bool pair) {
  constexpr bool X3 = three_parts(FMT), T2 = FMT == FMT_TF32X2, two = FMT == FMT_F16X2;
  return pair ? (two ? 1400 : 2050)
         : bn == 256 ? (X3 || T2 ? 2500 : two ? 1650 : 960)
         : bn == 128 ? (X3 || T2 ? 1500 : two ? 850 : 690)
                     : (T2 ? 1500 : X3 ? 900 : two ? 740 : 550);
}
constexpr int kWidths[3] = {256, 128, 64};
constexpr int width_index(int bn) { return bn == 256 ? 0 : bn == 128 ? 1 : 2; }

// How many CTAs share a tile, and the tile's width, for a GEMM of few tiles and a long contraction (the atoms' rows); `parts`
// is 1 if none should. A step of 32 columns takes about `clocks` however few tiles there are (see the head of this file), so
// K is shared out as far as the SMs go; handing the sums over costs 4000 clocks and more with the tile's width. Clusters do
// not fill every SM, those of eight hardly two thirds (96 fit, 112 took a second round).
// FMT_F16X3, whose rows' bits must not depend on how many there are, adds its pieces in K's order either way, and so is
// shared by as many CTAs as it has pieces, or not at all. From K = 1024 on: below that there is little to share, and GEMMs
// over a few thousand tokens, whose row count moves, stay out of it.
// Measured, recorded passes, whole -> shared: FMT_F16X2 648 x 1024 x 4096 47.5 us -> 28.2 (256 wide, 4 CTAs), 648 x 256 x 1024
// 14.2 -> 10.7 (128, 4); FMT_F16X3 21 x 512 x 2048 28.0 -> 12.0 (64, 4), 648 x 1024 x 4096 65.6 -> 44.3 (256, 4).
template <int FMT>
Plan plan_split(const GemmArgs& a, int bn_whole, int sms) {
  constexpr bool X3 = three_parts(FMT);
  const int steps = (a.K + 31) / 32, rows = cdiv(a.M, TBM);
  Plan best;
  if (a.K < 1024 || a.K % 32 || a.N % 64 || a.rms != 0.f) return best;
  if (rows * cdiv(a.N, bn_whole) > sms) return best;
  best.clocks = (long long) steps * step_clocks<FMT>(width_index(bn_whole));
  for (int i = 0; i < 3; ++i)
    for (int parts = 2; parts <= 8; parts *= 2) {
      if (a.N % kWidths[i] || kWidths[i] / parts < (X3 ? 16 : 32) || steps % parts || steps / parts < 4) continue;
      if (X3 && parts != (a.K <= 1024 ? 1 : a.K <= 4096 ? 4 : cdiv(a.K, 1024))) continue;
      if ((long long) rows * (a.N / kWidths[i]) * parts > (parts == 8 ? sms * 2 / 3 : sms * 7 / 8)) continue;
      const long long cost = (long long) (steps / parts) * step_clocks<FMT>(i) + 4000 + 55 * kWidths[i];
      if (cost < best.clocks) best.bn = kWidths[i], best.parts = parts, best.clocks = cost;
    }
  return best;
}

// One GEMM by itself.
template <int EPI, int FMT>
Plan plan_one(const GemmArgs& a, int sms) {
  // The tile width that finishes first. A tile's time per step of K goes with the shared-memory wavefronts it needs
  // (operand reads, fills, the converter, its share of the epilogue), which a narrower tile needs fewer of per tile
  // and more of per output column; the launch takes as many rounds as its fullest CTA has tiles. The token GEMMs
  // (thousands of row tiles) come out at 256; a GEMM over the atoms' rows (14 row tiles at 1728 atoms) at whatever
  // gives one round: 64 for 256 columns, 128 for 1024, 256 for 2048.
  const long long mt = cdiv(a.M, TBM);
  constexpr bool twelve = three_parts(FMT) || FMT == FMT_TF32X2;  // twelve bytes of operand reads per value and tile side
  constexpr int wavefronts[3] = {twelve ? 608 : FMT == FMT_F16X2 ? 416 : 272, twelve ? 408 : FMT == FMT_F16X2 ? 280 : 184,
                                 twelve ? 308 : FMT == FMT_F16X2 ? 212 : 140};
  Plan p;
  long long best = 0;
  for (int i = 0; i < 3; ++i) {
    if (a.N % kWidths[i] != 0) continue;
    const long long tiles = mt * (a.N / kWidths[i]), rounds = (tiles + sms - 1) / sms;
    if (p.bn == 0 || rounds * wavefronts[i] < best) p.bn = kWidths[i], best = rounds * wavefronts[i];
  }
  if (p.bn == 0) p.bn = a.N <= 64 ? 64 : 128;  // ragged widths: a tile with a zero-filled edge
  // A pair of CTAs per 256-row tile halves what each reads and stages of the weight. It pays in the formats of two and three
  // parts, whose weight tiles are the larger share (122138 rows: FMT_F16X3 w_in backward 258 us against 307, SwiGLU 353
  // against 383; FMT_F16X2 215 against 274, plain 56 against 60), once there is a tile for every pair of SMs; the formats of
  // one part are near HBM's rate without it, and the second CTA's signals make a step longer (SwiGLU 180 us against 164).
  constexpr bool kPair = three_parts(FMT) || FMT == FMT_F16X2 || FMT == FMT_TF32X2;
  p.pair = kPair && p.bn == 256 && cdiv(a.M, 2 * TBM) * (a.N / 256) >= sms / 2;
  if (EPI == EPI_PLAIN && !p.pair) {
    const Plan sp = plan_split<FMT>(a, p.bn, sms);
    if (sp.parts > 1) return sp;
  }
  return p;
}
template <int FMT>
long long clocks_of(const GemmArgs& a, const Plan& p, int sms) {
  const long long steps = (a.K + 31) / 32, c = full_clocks<FMT>(p.bn, p.pair);
  if (p.parts > 1) return steps / p.parts * step_clocks<FMT>(width_index(p.bn)) + 4000 + 55 * p.bn;
  const long long tiles = (long long) cdiv(a.M, p.pair ? 2 * TBM : TBM) * cdiv(a.N, p.bn), workers = p.pair ? sms / 2 : sms;
  return (tiles + workers - 1) / workers * steps * c;
}

// Two GEMMs as one launch, if that is expected to end before one after the other does; else bn is 0. A launch by itself costs
// 4-5 us (its start, the first tile on its way, the last one leaving). The clocks of a cut are those of the worker with most to do:
// where the atoms' tiles are so long that they outlast the rest, the two stay apart (1791 atoms, FMT_F16, backward of w_in with 128 steps
// a tile: 105 us apart, 118 together on tiles of 128 columns).
template <int EPI, int FMT>
Plan plan_two(const GemmArgs& a, const GemmArgs& b, int sms) {
  constexpr bool X3 = three_parts(FMT), kPair = X3 || FMT == FMT_F16X2 || FMT == FMT_TF32X2;
  Plan best;
  best.clocks = clocks_of<FMT>(a, plan_one<EPI, FMT>(a, sms), sms) + clocks_of<FMT>(b, plan_one<EPI, FMT>(b, sms), sms) + 8000;
  const long long sa = (a.K + 31) / 32, sb = (b.K + 31) / 32;
  for (int i = 0; i < 3; ++i) {
    const int bn = kWidths[i];
    if (a.N % bn || b.N % bn) continue;
    for (int pair = 0; pair <= (kPair && i == 0 ? 1 : 0); ++pair) {
      const long long ca = sa * full_clocks<FMT>(bn, pair), cb = sb * full_clocks<FMT>(bn, pair);
      const int rows = pair ? 2 * TBM : TBM;
      const int n0 = cdiv(a.M, rows) * (a.N / bn), n1 = cdiv(b.M, rows) * (b.N / bn), workers = std::min(pair ? sms / 2 : sms, n0 + n1);
      const int rounds = int(std::max(1LL, (ca + cb / 2) / cb));
      if (pair && n0 + n1 < sms / 2) continue;
      const Walk w(workers, n0, n1, rounds);
      long long most = 0;
      for (int who : {0, w.lead, workers - 1}) {  // the first with and without a tile of side 0's last round, the last
        const int own = w.full + (who < w.lead);
        int side, t, k = own, hi = own + n1 + 1;
        while (k < hi) {  // how many tiles it has
          const int mid = (k + hi) / 2;
          if (w.at(who, mid, side, t)) k = mid + 1;
          else hi = mid;
        }
        most = std::max(most, own * ca + (k - own) * cb);
      }
      // The SwiGLU epilogues of three parts, whose arguments come through an index, take 11-13 % longer, and leave the issuer waiting:
      // 1728 atoms, forward, 394 us apart, 427 together; 648 atoms 130 and 124.
      if (X3 && (EPI == EPI_SWIGLU || EPI == EPI_SWIGLU_BWD)) most += most / 4;
      if (most < best.clocks) best.bn = bn, best.pair = pair, best.parts = 1, best.rounds = rounds, best.clocks = most;
    }
    if (EPI != EPI_PLAIN || bn != 64 || a.K < 1024 || a.K % 32 || a.rms != 0.f || b.rms != 0.f || (X3 && b.K > 1024)) continue;
    for (int parts = 2; parts <= 8; parts *= 2) {  // side 0's tiles shared as plan_split would (few rows: narrow tiles)
      if (bn / parts < (X3 ? 16 : 32) || sa % parts || sa / parts < 4) continue;
      if (X3 && parts != (a.K <= 1024 ? 1 : a.K <= 4096 ? 4 : cdiv(a.K, 1024))) continue;
      const long long ctas = ((long long) cdiv(a.M, TBM) * (a.N / bn) + cdiv((long long) cdiv(b.M, TBM) * (b.N / bn), parts)) * parts;
      if (ctas > (parts == 8 ? sms * 2 / 3 : sms * 7 / 8)) continue;
      const long long cost = std::max(sa / parts, sb) * step_clocks<FMT>(i) + 4000 + 55 * bn;
      if (cost < best.clocks) best.bn = bn, best.pair = false, best.parts = parts, best.clocks = cost;
    }
  }
  return best;
}

template <int EPI, int FMT, int SIDES>
void launch_plan(Stream& st, const GemmTask* q, const Plan& p) {
  constexpr bool kPair = three_parts(FMT) || FMT == FMT_F16X2 || FMT == FMT_TF32X2;
  if constexpr (kPair)
    if (p.pair) return launch_tc<EPI, 256, FMT, true, false, SIDES>(st, q, p);
  if constexpr (EPI == EPI_PLAIN)
    if (p.parts > 1) {
      if constexpr (SIDES == 1) {
        if (p.bn == 256) return launch_tc<EPI, 256, FMT, false, true, SIDES>(st, q, p);
        if (p.bn == 128) return launch_tc<EPI, 128, FMT, false, true, SIDES>(st, q, p);
      }
      return launch_tc<EPI, 64, FMT, false, true, SIDES>(st, q, p);
    }
  if (p.bn == 256) launch_tc<EPI, 256, FMT, false, false, SIDES>(st, q, p);
  else if (p.bn == 128) launch_tc<EPI, 128, FMT, false, false, SIDES>(st, q, p);
  else launch_tc<EPI, 64, FMT, false, false, SIDES>(st, q, p);
}

}  // namespace

template <int EPI, int FMT>
void run_format(Stream& st, const GemmTask* q, int n) {
  const int sms = tensor_state().sms;
  // (weights with spread values and the forward of a wide model in tf32 mode: always apart)
  if constexpr (EPI != EPI_COMPRESS && FMT != FMT_F16X3_FULL && FMT != FMT_TF32)
    if (n == 2) {
      const bool alike = EPI != EPI_PLAIN || !q[0].a.res == !q[1].a.res;
      const Plan p = alike ? plan_two<EPI, FMT>(q[0].a, q[1].a, sms) : Plan{};
      if (p.bn) return launch_plan<EPI, FMT, 2>(st, q, p);
    }
  for (int i = 0; i < n; ++i) launch_plan<EPI, FMT, 1>(st, q + i, plan_one<EPI, FMT>(q[i].a, sms));
}
// the plain epilogue's instances are two files' work (gemm_tc_plain_x3.cu)
extern template void run_format<EPI_PLAIN, FMT_F16X3>(Stream&, const GemmTask*, int);
extern template void run_format<EPI_PLAIN, FMT_F16X3_FULL>(Stream&, const GemmTask*, int);

template <int EPI>
void run_tensor(Stream& st, const GemmTask* q, int n) {
  for (int i = 0; i < n; ++i)
    if (q[i].a.rms != 0.f && ((EPI != EPI_PLAIN && EPI != EPI_SWIGLU) || (!three_parts(q[i].w.fmt) && q[i].w.fmt != FMT_F16X2 && q[i].w.fmt != FMT_TF32X2)))
      throw Error(3, "gemm: no kernel for this operand format and epilogue after a norm");
  switch (q[0].w.fmt) {
    case FMT_F16X3: return run_format<EPI, FMT_F16X3>(st, q, n);
    case FMT_F16X3_FULL: return run_format<EPI, FMT_F16X3_FULL>(st, q, n);
    case FMT_F16X2: return run_format<EPI, FMT_F16X2>(st, q, n);
    case FMT_F16: return run_format<EPI, FMT_F16>(st, q, n);
    case FMT_BF16: return run_format<EPI, FMT_BF16>(st, q, n);
    default: break;
  }
  // the tf32 formats: the forward of wide models (Model::put_mat)
  if constexpr (EPI != EPI_SILU_BWD && EPI != EPI_SWIGLU_BWD) {
    if (q[0].w.fmt == FMT_TF32X2) return run_format<EPI, FMT_TF32X2>(st, q, n);
    if (q[0].w.fmt == FMT_TF32) return run_format<EPI, FMT_TF32>(st, q, n);
  }
  throw Error(3, "gemm: no kernel for this operand format and epilogue");
}

}  // namespace petb
