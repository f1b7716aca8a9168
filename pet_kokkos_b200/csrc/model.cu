// The PET network: see model.h.
#include "model.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "../../include/pet_b200.h"
#include "attention.h"
#include "gemm.h"

namespace petb {

using Taps = std::map<std::string, std::pair<const float*, size_t>>;

// ---- weights -----------------------------------------------------------------
//
// A checkpoint tensor is uploaded once as it is stored (doubles) and every layout the kernels read is made from it
// on the device: fp32, and both orientations packed in the formats the calculator's GEMM mode reads (gemm.h). The
// SwiGLU row pairing and the fold of compress.0 are index maps and short fp64 sums over the uploaded tensors, so
// the host never loops over a weight.

namespace {

// Row a of the prepared matrix comes from this row of the stored one. A SwiGLU input layer is stored as [v ; g]
// (F value rows, then F gate rows) and read as (v_0, g_0, v_1, g_1, ...) so that a gate pair meets in one GEMM
// thread's run of columns (the reference does the same at load, src/model.cpp:211-222).
__device__ __forceinline__ int stored_row(int a, int rows, int paired) { return paired ? (a & 1) * (rows / 2) + (a >> 1) : a; }

// src [rows, ld] doubles (the first `cols` columns of each row) -> [rows, cols] floats.
// Times gain[column], unless null.
__global__ void k_weight_rows(const double* src, int ld, int rows, int cols, int paired, const double* gain, float* out) {
  const size_t n = size_t(rows) * cols, i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int a = int(i / cols), b = int(i % cols);
  const double x = src[size_t(stored_row(a, rows, paired)) * ld + b];
  out[i] = float(gain ? x * gain[b] : x);
}
__global__ void k_weight_vector(const double* src, int len, int paired, float* out) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < len) out[a] = float(src[stored_row(a, len, paired)]);
}

// compress.0 acts on [edge embedding of (v, |v|) | species embedding | input_edge]; the first two blocks are linear
// in four numbers and in a table row, so their products with compress.0 are formed once, in fp64 with every product
// and sum rounded on its own, in column order (the reference's fold, src/model.cpp:233-254, gives the same bits):
//   wx[d, c]  = sum_j W[d, j] We[j, c]        b[d] = b0[d] + sum_j W[d, j] be[j]
//   tab[s, d] = sum_j T[s, j] W[d, D + j]
__global__ void k_fold_geometry(const double* W, int K, const double* We, const double* be, const double* b0, int D, double* wx,
                                double* b) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= D) return;
  double x[4] = {0.0, 0.0, 0.0, 0.0}, bias = b0[d];
  for (int j = 0; j < D; ++j) {
    const double w = W[size_t(d) * K + j];
    for (int c = 0; c < 4; ++c) x[c] = __dadd_rn(x[c], __dmul_rn(w, We[j * 4 + c]));
    bias = __dadd_rn(bias, __dmul_rn(w, be[j]));
  }
  for (int c = 0; c < 4; ++c) wx[d * 4 + c] = x[c];
  b[d] = bias;
}
__global__ void k_fold_species(const double* W, int K, const double* T, int ns, int D, double* tab) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ns * D) return;
  const int s = i / D, d = i % D;
  double acc = 0.0;
  for (int j = 0; j < D; ++j) acc = __dadd_rn(acc, __dmul_rn(T[size_t(s) * D + j], W[size_t(d) * K + D + j]));
  tab[i] = acc;
}

// W = A . B and b = A . x + y, what two linear layers without anything between them come to. In fp64.
__global__ void k_fold_layers(const double* A, const double* B, const double* x, const double* y, int rows, int inner, int cols, double* W, double* b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * (cols + 1)) return;
  const int r = i / (cols + 1), c = i % (cols + 1);
  double acc = c < cols ? 0.0 : y[r];
  for (int j = 0; j < inner; ++j) acc += A[size_t(r) * inner + j] * (c < cols ? B[size_t(j) * cols + c] : x[j]);
  if (c < cols) W[size_t(r) * cols + c] = acc;
  else b[r] = acc;
}

// A tensor's doubles on the device for the duration of the load.
struct Staged {
  double* p = nullptr;
  int rows = 0, cols = 0;
  explicit Staged(const Tensor& t) {
    rows = t.shape.empty() ? 1 : int(t.dim(0));
    cols = t.shape.size() > 1 ? int(t.dim(1)) : 1;
    alloc(t.data.size());
    PETB_CUDA(cudaMemcpy(p, t.data.data(), t.data.size() * sizeof(double), cudaMemcpyHostToDevice));
  }
  explicit Staged(size_t n) { alloc(n); }
  ~Staged() { cudaFree(p); }
  Staged(const Staged&) = delete;
  void alloc(size_t n) { PETB_CUDA(cudaMalloc(&p, (n ? n : 1) * sizeof(double))); }
};

// What the network reads from a checkpoint, as (tensor name, how it is prepared).
enum class Prep { Table, Matrix, Vector, PairedMatrix, PairedVector, CompressFold, ExpansionFold };  // Table: read row by row, never a GEMM operand
struct PlanItem {
  std::string name;
  Prep prep;
  int layer = 0;
  std::string gain;  // an RMSNorm's weight that the matrix takes with it: the norm before it is then the row's 1 / rms alone
};

std::vector<PlanItem> weight_plan(const Hypers& h, bool gains) {
  std::vector<PlanItem> plan;
  const bool ff = h.feedforward, paired = h.swiglu;
  auto dense = [&](const std::string& stem, bool pair_rows = false, const std::string& gain = "") {
    plan.push_back({stem + ".weight", pair_rows ? Prep::PairedMatrix : Prep::Matrix, 0, gain});
    plan.push_back({stem + ".bias", pair_rows ? Prep::PairedVector : Prep::Vector});
  };
  auto norm = [&](const std::string& stem) {
    plan.push_back({stem + ".weight", Prep::Vector});
    if (h.layernorm) plan.push_back({stem + ".bias", Prep::Vector});
  };
  // a layer and the norm before it
  auto normed = [&](const std::string& stem, bool pair_rows, const std::string& before) {
    dense(stem, pair_rows, gains ? before + ".weight" : "");
    if (!gains) norm(before);
  };
  plan.push_back({"edge_embedder.weight", Prep::Table});
  for (int L = 0; L < h.num_gnn_layers; ++L) {
    const std::string layer = "gnn_layers." + std::to_string(L);
    plan.push_back({layer + ".compress.0", Prep::CompressFold, L});
    dense(layer + ".compress.2");
    for (int a = 0; a < h.num_attention_layers; ++a) {
      const std::string block = layer + ".trans.layers." + std::to_string(a);
      for (const char* part : {".attention.output_linear", ".mlp.w_out"}) dense(block + part);
      normed(block + ".attention.input_linear", false, block + ".norm_attention");
      normed(block + ".mlp.w_in", paired, block + ".norm_mlp");
      if (!h.expanded_node()) continue;
      for (const char* part : {".center_contraction", ".center_mlp.w_out"}) dense(block + part);
      plan.push_back({block, Prep::ExpansionFold});
      normed(block + ".center_mlp.w_in", paired, block + ".norm_center_features");
    }
    if (ff) {
      const std::string n = "combination_norms." + std::to_string(L), m = "combination_mlps." + std::to_string(L);
      plan.push_back({n + ".weight", Prep::Vector}), plan.push_back({n + ".bias", Prep::Vector});
      dense(m + ".0"), dense(m + ".2");
    }
  }
  for (int i = 0; i < h.num_readout_layers; ++i) {
    const std::string r = std::to_string(i);
    plan.push_back({"node_embedders." + r + ".weight", Prep::Table});
    for (const char* side : {"node", "edge"}) {
      dense(std::string(side) + "_heads.energy." + r + ".0"), dense(std::string(side) + "_heads.energy." + r + ".2");
      const std::string last = std::string(side) + "_last_layers.energy." + r + ".energy___0";
      plan.push_back({last + ".weight", Prep::Table}), plan.push_back({last + ".bias", Prep::Vector});
    }
  }
  return plan;
}

// Whether a gain damps some features by 2^-12 and more against others (zeros leave nothing to damp). Their values may stand out by as
// much, and a row's scale is that of its largest: two parts hold 22 bits down to 2^-18 of it.
bool damps(const Tensor& gain) {
  double least = INFINITY, most = 0.0;
  for (double g : gain.data)
    if (g != 0.0) least = std::min(least, std::fabs(g)), most = std::max(most, std::fabs(g));
  return least < most / 4096.0;
}

}  // namespace

void Model::put_mat(const std::string& name, const double* src, int ld, int rows, int cols, bool paired, bool operand, const double* gain) {
  const size_t n = size_t(rows) * cols;
  float* dev = nullptr;
  PETB_CUDA(cudaMalloc(&dev, (n + 4) * sizeof(float)));
  owned_.push_back(dev);
  if (n) k_weight_rows<<<cdiv((long long) n, 256), 256>>>(src, ld, rows, cols, paired ? 1 : 0, gain, dev);
  PETB_CUDA(cudaGetLastError());
  Mat m;
  m.w = dev, m.rows = rows, m.cols = cols;
  if (operand) {  // both orientations in the native format (every mode runs its smallest GEMMs in it) and in the mode's own
    auto pack = [&](Format f, bool transposed) {
      const int r = transposed ? cols : rows, k = transposed ? rows : cols;
      uint16_t* out = nullptr;
      const size_t bytes = (packed_halves(f, r, k) * 2 + 15) & ~size_t(15);
      PETB_CUDA(cudaMalloc(&out, bytes + 2 * unscale_halves(r)));
      owned_.push_back(out);
      return pack_weight(nullptr, f, dev, transposed ? 1 : cols, transposed ? cols : 1, r, k, out,
                         reinterpret_cast<uint16_t*>(reinterpret_cast<char*>(out) + bytes));
    };
    // At widths past 256 the forward of the 3xTF32 and tf32 modes keeps the tf32 instructions. The accumulator's
    // truncations pull every product sum toward zero by a factor that goes with their number, one per 8 columns of K and
    // product there, one per 16 in fp16; and where activations are truncated to 11 bits, the last bit of a sum decides some
    // of them. Up to 256 columns energies agree between the two to 1e-6 (3xTF32) and 2e-4 (tf32); at 512, where a network
    // energy of 2.6 eV per atom stood against -2.6 of composition energy, to 2e-4 and 2e-3 of their sum: there the modes'
    // energies stay what they were. Forces feel neither, so the backward runs in fp16 parts at every width.
    const Format fmt = format_of(mode_), wide_forward = fmt == FMT_F16X2 ? FMT_TF32X2 : fmt == FMT_F16 ? FMT_TF32 : fmt;
    const Format forward = wide() ? wide_forward : fmt;
    m.nat = pack(FMT_F16X3, false), m.nat_t = pack(FMT_F16X3, true);
    m.fast = forward == FMT_F16X3 ? m.nat : pack(forward, false);
    m.fast_t = fmt == FMT_F16X3 ? m.nat_t : pack(fmt, true);
  }
  mat_[name] = m;
}

// A weight and its norm's gain in one, or false and nothing kept. In the native mode the norm stays by itself where the gain would set the
// weight's columns so far apart that its format needs eight products instead of six, which also never share a launch. One gain of 2^-6,
// one way -> the other, each against all gains near one: 21 atoms 1.033 -> 1.01-1.03, water648 1.024 -> 1.01-1.02, diamond1728 both 1.02.
// 3xTF32 has three products either way, and folds any but gains that damp by more than its parts have to spare.
bool Model::put_after_norm(const std::string& name, const double* src, int rows, int cols, bool paired, const double* gain, const Tensor& host_gain) {
  if (mode_ != GEMM_NATIVE && damps(host_gain)) return false;
  const size_t kept = owned_.size();
  put_mat(name, src, cols, rows, cols, paired, true, gain);
  PETB_CUDA(cudaDeviceSynchronize());
  Mat& m = mat_[name];
  if (mode_ != GEMM_NATIVE || !values_spread(m.nat, rows)) return m.after_norm = true;
  for (; owned_.size() > kept; owned_.pop_back()) cudaFree(owned_.back());
  mat_.erase(name);
  return false;
}

void Model::put_vec(const std::string& name, const double* src, int len, bool paired) {
  float* dev = nullptr;
  PETB_CUDA(cudaMalloc(&dev, (len > 0 ? len : 1) * sizeof(float)));
  owned_.push_back(dev);
  if (len) k_weight_vector<<<cdiv(len, 256), 256>>>(src, len, paired ? 1 : 0, dev);
  PETB_CUDA(cudaGetLastError());
  vec_[name] = dev;
}

const Mat& Model::mat(const std::string& name) const {
  auto it = mat_.find(name);
  if (it == mat_.end()) throw Error(1, "model: missing matrix '" + name + "'");
  return it->second;
}
const float* Model::vec(const std::string& name) const {
  auto it = vec_.find(name);
  if (it == vec_.end()) throw Error(1, "model: missing vector '" + name + "'");
  return it->second;
}

// compress.0 of layer L -> "@x4" [D,4], "@b" [D], "@tab" [n_species, D] and, past the first layer, "@in" [D,D] (the
// block that still multiplies input_edge). At layer 0 the species block is the edge embedder's table itself.
void Model::fold_compress(const Checkpoint& ck, const std::string& c0, int L) {
  const std::string layer = "gnn_layers." + std::to_string(L);
  const Staged W(ck.at(c0 + ".weight")), b0(ck.at(c0 + ".bias"));
  const Staged We(ck.at(layer + ".edge_embedder.weight")), be(ck.at(layer + ".edge_embedder.bias"));
  const Staged T(ck.at(L == 0 ? "edge_embedder.weight" : layer + ".neighbor_embedder.weight"));
  const int D = W.rows, K = W.cols, ns = T.rows;
  if (K != (L == 0 ? 2 : 3) * D || T.cols != D || We.rows != D || We.cols != 4)
    throw Error(1, "model: '" + c0 + "' does not have the shape of a compress layer");
  const size_t nx = size_t(D) * 4, nb = size_t(D), nt = size_t(ns) * D;
  const Staged wx(nx), b(nb), tab(nt);
  k_fold_geometry<<<cdiv(D, 128), 128>>>(W.p, K, We.p, be.p, b0.p, D, wx.p, b.p);
  k_fold_species<<<cdiv((long long) ns * D, 128), 128>>>(W.p, K, T.p, ns, D, tab.p);
  PETB_CUDA(cudaGetLastError());
  put_mat(c0 + "@x4", wx.p, 4, D, 4, false, false);
  put_vec(c0 + "@b", b.p, D, false);
  put_mat(c0 + "@tab", tab.p, D, ns, D, false, false);
  if (L > 0) put_mat(c0 + "@in", W.p + 2 * D, K, D, D, false, true);
  PETB_CUDA(cudaDeviceSynchronize());  // the staged tensors are freed on return
}

// A block's expansion of the atoms' rows of the attention's output, with the output layer before it: nothing else reads those rows.
// "@expand" [d_node, d_pet], "@expand_b". Two GEMMs on the atoms' chain become one, beside the edges' output layer.
void Model::fold_expansion(const Checkpoint& ck, const std::string& block) {
  const Staged A(ck.at(block + ".center_expansion.weight")), y(ck.at(block + ".center_expansion.bias"));
  const Staged B(ck.at(block + ".attention.output_linear.weight")), x(ck.at(block + ".attention.output_linear.bias"));
  if (A.cols != B.rows || x.rows < B.rows || y.rows < A.rows)  // (the fold reads them at these lengths)
    throw Error(1, "model: '" + block + ".center_expansion' does not have the shape of an expansion");
  const Staged W(size_t(A.rows) * B.cols), b(size_t(A.rows));
  k_fold_layers<<<cdiv((long long) A.rows * (B.cols + 1), 128), 128>>>(A.p, B.p, x.p, y.p, A.rows, A.cols, B.cols, W.p, b.p);
  PETB_CUDA(cudaGetLastError());
  put_mat(block + "@expand", W.p, B.cols, A.rows, B.cols, false, true);
  put_vec(block + "@expand_b", b.p, A.rows, false);
  PETB_CUDA(cudaDeviceSynchronize());  // the staged tensors are freed on return
}

Model::Model(const Checkpoint& ck, int gemm_mode) : h_(ck.hypers), scale_(ck.energy_scale), mode_(gemm_mode) {
  const bool ff = h_.feedforward, ln = h_.layernorm, expanded = h_.expanded_node(), swiglu = h_.swiglu;

  // The two families the reference implements (src/model.cpp:314-334); anything else is refused by name.
  if (ff && (!h_.preln || ln || !swiglu || !expanded))
    throw Error(1, "model: the feedforward featurizer needs PreLN + RMSNorm + SwiGLU with d_node != d_pet");
  if (!ff && (h_.preln || !ln || swiglu || expanded))
    throw Error(1, "model: the residual featurizer needs PostLN + LayerNorm + SiLU with d_node == d_pet");
  if (h_.num_attention_layers < 1) throw Error(1, "model: num_attention_layers must be >= 1");
  if (h_.head_dim * h_.num_heads != h_.d_pet) throw Error(1, "model: num_heads * head_dim must equal d_pet");
  if (h_.d_pet % 4 || h_.d_node % 4 || h_.d_head % 4 || h_.d_feedforward % 4)
    throw Error(1, "model: layer widths must be multiples of 4");

  for (const PlanItem& it : weight_plan(h_, folds_norms())) {
    if (it.prep == Prep::CompressFold) {
      fold_compress(ck, it.name, it.layer);
      continue;
    }
    if (it.prep == Prep::ExpansionFold) {
      fold_expansion(ck, it.name);
      continue;
    }
    const Tensor& t = ck.at(it.name);
    const bool matrix = it.prep == Prep::Table || it.prep == Prep::Matrix || it.prep == Prep::PairedMatrix;
    const bool paired = it.prep == Prep::PairedMatrix || it.prep == Prep::PairedVector;
    if (matrix && t.shape.size() != 2) throw Error(1, "model: expected a 2-D tensor '" + it.name + "'");
    const Staged dev(t);
    if (!it.gain.empty()) {
      const Staged gain(ck.at(it.gain));
      if (gain.rows * gain.cols != dev.cols) throw Error(1, "model: '" + it.gain + "' does not have the width of the layer after it");
      if (!put_after_norm(it.name, dev.p, dev.rows, dev.cols, paired, gain.p, ck.at(it.gain))) {
        put_mat(it.name, dev.p, dev.cols, dev.rows, dev.cols, paired, true);
        put_vec(it.gain, gain.p, dev.cols, false);
        norms_apart_ = true;
      }
      PETB_CUDA(cudaDeviceSynchronize());  // before the gain goes
    } else if (matrix) put_mat(it.name, dev.p, dev.cols, dev.rows, dev.cols, paired, it.prep != Prep::Table);
    else put_vec(it.name, dev.p, int(t.numel()), paired);
    PETB_CUDA(cudaDeviceSynchronize());
  }
  const size_t ns = ck.composition_energies.size();
  PETB_CUDA(cudaMalloc(&comp_, (ns ? ns : 1) * sizeof(double)));
  PETB_CUDA(cudaMemcpy(comp_, ck.composition_energies.data(), ns * sizeof(double), cudaMemcpyHostToDevice));
  if (h_.adaptive() && !h_.adaptive_solver) {  // from 0.5 A to the cutoff, a quarter of the taper width apart
    std::vector<double> probes;
    for (double r = 0.5; r < h_.cutoff - 1e-12; r += h_.cutoff_width_adaptive / 4.0) probes.push_back(r);
    n_probes_ = int(probes.size());
    PETB_CUDA(cudaMalloc(&probes_, (probes.size() ? probes.size() : 1) * sizeof(double)));
    PETB_CUDA(cudaMemcpy(probes_, probes.data(), probes.size() * sizeof(double), cudaMemcpyHostToDevice));
  }
  PETB_CUDA(cudaDeviceSynchronize());
  for (auto& [name, m] : mat_)
    if (m.nat.main) {
      full_if_spread(m.nat, m.rows), full_if_spread(m.nat_t, m.cols);
      if (m.fast.fmt == FMT_F16X3) m.fast = m.nat;
      if (m.fast_t.fmt == FMT_F16X3) m.fast_t = m.nat_t;
    }
  // a blocking copy from pageable memory returns once staged: fence, since the evaluations run on a stream that
  // does not wait for the legacy one
  PETB_CUDA(cudaDeviceSynchronize());
}

Model::~Model() {
  for (void* p : owned_) cudaFree(p);
  cudaFree(comp_);
  cudaFree(probes_);
}

// ---- the GEMM calls, by role ------------------------------------------------------

namespace {

// The attention mode that goes with a GEMM mode unless PET_ATTN names one (native | tf32x3 | tf32), as the reference's
// Options::attention / PET_ATTN (include/pet/calculator.hpp:46-49): Native with native GEMMs, TF32x3 with 3xTF32 GEMMs,
// and the single-pass TF32 form with the tf32 and bf16 speed modes.
int attention_mode_for(int gemm_mode) {
  static const int forced = [] {
    const char* e = std::getenv("PET_ATTN");
    if (!e) return -1;
    const std::string v(e);
    return v == "native" ? int(ATTN_NATIVE) : (v == "tf32x3" || v == "3xtf32") ? int(ATTN_TF32X3) : v == "tf32" ? int(ATTN_TF32) : -1;
  }();
  if (forced >= 0) return forced;
  return gemm_mode == GEMM_NATIVE ? ATTN_NATIVE : gemm_mode == GEMM_TF32X3 ? ATTN_TF32X3 : ATTN_TF32;
}

// Rows of an activation or adjoint, with the bits of each row's largest magnitude where the mode's operand format wants
// them (gemm.h); whatever writes the rows keeps them.
struct Rows {
  float* p = nullptr;
  uint32_t* mx = nullptr;
  Rows from(size_t row, int ld) const { return {p + row * ld, mx ? mx + row : nullptr}; }
};

// The arrays of row maxima of one pass: one zeroed block from `save`, a fresh part of it for every tensor written (a GEMM
// raises its rows' maxima atomically, so they start from zero). Modes that need none get null pointers; so does whatever
// the block has no room left for (an edge MLP in very small chunks), whose GEMM then looks for the maxima itself.
class RowMaxima {
 public:
  RowMaxima(Stream& st, Arena& save, size_t words) : size_(words) {
    if (!words) return;
    base_ = save.alloc<uint32_t>(words);
    PETB_CUDA(cudaMemsetAsync(base_, 0, words * sizeof(uint32_t), st.s));
  }
  uint32_t* take(size_t rows) {
    rows = (rows + 31) & ~size_t(31);
    if (used_ + rows > size_) return nullptr;
    uint32_t* p = base_ + used_;
    used_ += rows;
    return p;
  }
  Rows fresh(float* p, size_t rows) { return {p, take(rows)}; }

 private:
  uint32_t* base_ = nullptr;
  size_t size_ = 0, used_ = 0;
};

struct Gemms {
  Stream& st;
  Arena& tmp;

  static GemmArgs args(const Rows& out, const Rows& in, const Mat& W, bool transposed, int M) {
    GemmArgs a;
    a.A = in.p, a.a_max = in.mx, a.C = out.p, a.c_max = out.mx, a.M = M;
    a.N = transposed ? W.cols : W.rows, a.K = transposed ? W.rows : W.cols;
    a.lda = a.K, a.ldc = a.ldr = a.ldp = a.N;
    a.nat = transposed ? W.nat_t : W.nat, a.fast = transposed ? W.fast_t : W.fast;
    return a;
  }
  // out[M, W.rows] = in[M, W.cols] . W^T + bias (+ res for rows >= res_row0)
  static GemmArgs linear_args(const Rows& out, const Rows& in, const Mat& W, const float* bias, int M, const float* res = nullptr,
                              int res_row0 = 0) {
    GemmArgs a = args(out, in, W, false, M);
    a.bias = bias, a.res = res, a.res_row0 = res_row0;
    return a;
  }
  // out = silu(pre), pre = in . W^T + bias, kept when `pre` is given
  static GemmArgs silu_args(const Rows& out, float* pre, const Rows& in, const Mat& W, const float* bias, int M) {
    GemmArgs a = args(out, in, W, false, M);
    a.bias = bias, a.pre = pre, a.epi = EPI_SILU;
    return a;
  }
  // pre[M, 2F] = in . W^T + bias (interleaved v, g); h[M, F] = v * sigmoid(g)
  static GemmArgs swiglu_args(const Rows& h, float* pre, const Rows& in, const Mat& W, const float* bias, int M) {
    GemmArgs a = args(h, in, W, false, M);
    a.ldc = W.rows / 2, a.bias = bias, a.pre = pre, a.epi = EPI_SWIGLU;
    return a;
  }
  // in_adj[M, W.cols] (+)= out_adj[M, W.rows] . W
  static GemmArgs linear_bwd_args(const Rows& in_adj, const Rows& out_adj, const Mat& W, int M, bool acc) {
    GemmArgs a = args(in_adj, out_adj, W, true, M);
    a.res = acc ? in_adj.p : nullptr;
    return a;
  }
  // grad[M, W.cols] = (out_adj . W) * silu'(pre)
  static GemmArgs silu_bwd_args(const Rows& grad, const Rows& out_adj, const Mat& W, const float* pre, int M) {
    GemmArgs a = args(grad, out_adj, W, true, M);
    a.pre = const_cast<float*>(pre), a.epi = EPI_SILU_BWD;
    return a;
  }
  // pre_adj[M, 2F] from h_adj = out_adj . W_out and the saved pre
  static GemmArgs swiglu_bwd_args(const Rows& pre_adj, const Rows& out_adj, const Mat& w_out, const float* pre, int M) {
    GemmArgs a = args(pre_adj, out_adj, w_out, true, M);
    a.ldc = a.ldp = 2 * w_out.cols, a.pre = const_cast<float*>(pre), a.epi = EPI_SWIGLU_BWD;
    return a;
  }
  void one(const GemmArgs& a) const { gemm(st, tmp, a); }
  // The atoms' GEMM and the edges' of one step.
  void two(const GemmArgs& atoms, const GemmArgs& edges) const { gemm_two(st, tmp, atoms, edges); }
  void linear(const Rows& out, const Rows& in, const Mat& W, const float* bias, int M, const float* res = nullptr, int res_row0 = 0) const {
    one(linear_args(out, in, W, bias, M, res, res_row0));
  }
  void linear_silu(const Rows& out, float* pre, const Rows& in, const Mat& W, const float* bias, int M) const {
    one(silu_args(out, pre, in, W, bias, M));
  }
  void swiglu_in(const Rows& h, float* pre, const Rows& in, const Mat& W, const float* bias, int M) const {
    one(swiglu_args(h, pre, in, W, bias, M));
  }
  void linear_bwd(const Rows& in_adj, const Rows& out_adj, const Mat& W, int M, bool acc) const { one(linear_bwd_args(in_adj, out_adj, W, M, acc)); }
  void linear_silu_bwd(const Rows& grad, const Rows& out_adj, const Mat& W, const float* pre, int M) const {
    one(silu_bwd_args(grad, out_adj, W, pre, M));
  }
  // act = silu(pre), pre = in . W_in^T + b + tab[species] + wx . (v, |v|): compress.0 past the first layer
  void compress(const Rows& act, float* pre, const Rows& in, const Mat& W, const float* b, const Mat& tab, const Mat& x4,
                const PackedEdges& pk) const {
    GemmArgs a = args(act, in, W, false, pk.E);
    a.bias = b, a.pre = pre, a.tab = tab.w, a.sp = pk.species, a.wx = x4.w, a.vec = pk.vec, a.dist = pk.dist, a.epi = EPI_COMPRESS;
    gemm(st, tmp, a);
  }
};

// One swap of rows with the other ranks (Exchange::edges, include/pet/exchange.hpp:36-40): out[n_live, width] goes to
// the ranks that own the ghosts, in[n_live, width] comes back with the partner edges' rows. Every rank calls it the same
// number of times, with or without live edges of its own.
void exchange_rows(Stream& st, const PackedEdges& pk, const float* out, float* in, int width) {
  const pet_exchange* ex = static_cast<const pet_exchange*>(pk.exchange);
  if (!ex || !ex->edges) throw Error(3, "pet: an exchanged list without an edges() callback");
  if (ex->edges(ex->user, out, in, pk.n_live, width, static_cast<void*>(st.s)) != 0)
    throw Error(1, "pet: the exchange's edges() failed");
  order_after_legacy_stream(st);
}

struct Scope {
  Arena& a;
  Arena::Mark m;
  explicit Scope(Arena& ar) : a(ar), m(ar.mark()) {}
  ~Scope() { a.rewind(m); }
};

void tap(Taps* taps, const std::string& name, const float* p, size_t n) {
  if (taps) (*taps)[name] = {p, n};
}

}  // namespace

// ---- the tail shared by both featurizers ------------------------------------------

PassOut Model::finish(Stream& st, Arena& save, const PackedEdges& pk, bool grad, float* x4_adj, const float* cutoff_adj,
                      float* cf_adj, double* per_atom) {
  PassOut out;
  out.per_atom = per_atom;
  out.f.energy = save.alloc<double>(pk.B);
  if (!grad) {
    const ProfScope ps(st, PC_FORCES, 0.0, 8.0 * pk.B);
    structure_sums(st, out.f.energy, nullptr, per_atom, nullptr, pk.soff, pk.B);
    return out;
  }
  out.has_forces = true;
  out.f.edge_grad = save.alloc<double>(3 * size_t(pk.E > 0 ? pk.E : 1));
  out.f.forces = save.alloc<double>(3 * size_t(pk.n_atoms));
  out.f.vir_atom = save.alloc<double>(9 * size_t(pk.n_atoms));
  out.f.vir6 = save.alloc<double>(6 * size_t(pk.B));
  forces_and_virial(st, save, out.f, pk, x4_adj, cutoff_adj, cf_adj, cutoff_spec(), scale_, out.f.energy, per_atom);
  return out;
}

PassOut Model::run(Stream& st, Arena& save, Arena& tmp, const PackedEdges& pk, bool grad, int mode, Taps* taps,
                   const RunOptions& opt) {
  if (h_.feedforward) return run_feedforward(st, save, tmp, pk, grad, mode, taps, opt);
  last_tier_ = RECOMPUTE_NEVER, last_estimate_ = 0;
  return run_residual(st, save, tmp, pk, grad, mode, taps);
}

// ---- the feedforward featurizer ---------------------------------------------------
//
// How much of the forward the backward keeps (the reference's Recompute tiers, include/pet/config.hpp:19-24,
// src/feedforward.cpp:355-420): Never keeps every saved activation; Wide drops the two widest per block (the
// attention's qkv [T,3D] and the edge MLP's pre-activation [E,2F]) and rebuilds them in the backward with one norm and
// one GEMM each; Layers also keeps only each layer's inputs and re-runs one layer's forward at a time in the
// backward. Under Wide and Layers the edge MLP runs a chunk of edge rows at a time, forward and backward, so its wide
// temporaries are a chunk's. A row's GEMM result does not depend on which rows share its launch, so in the native
// mode every tier gives the bits of Never.

int Model::edge_chunk_rows(int E) {
  if (const char* c = std::getenv("PET_EDGE_CHUNK"))
    if (std::atoi(c) > 0) return std::atoi(c);
  const int eighth = (E + 7) / 8;
  return eighth > 65536 ? eighth : 65536;  // an eighth of the edges, never so few rows that the GEMMs run short
}

// Bytes the two pools hold at their fullest during one feedforward evaluation with forces under a tier: the sums of
// what run_feedforward takes from `save` and the largest of its scopes of `tmp`, from the shapes; 3 % and a few MiB on
// top for the pools' 256-byte rounding and the small per-atom and per-structure arrays of the force fold.
MemoryNeed Model::memory_need(int tier, int N, int E, int n_live) const {
  MemoryNeed need;
  if (!h_.feedforward) return need;
  const double D = h_.d_pet, H = h_.num_heads, F = h_.d_feedforward, Dn = h_.d_node, Dh = h_.d_head;
  const double G = h_.num_gnn_layers, A = h_.num_attention_layers;
  const double n = N, e = E, T = n + e, live = n_live;
  const bool keep = tier == RECOMPUTE_NEVER, relayer = tier == RECOMPUTE_LAYERS;
  const double c = keep ? e : std::min(e, double(edge_chunk_rows(E)));
  // save: what lives for the whole pass
  double save = (G + 1) * n * Dn + e * D + G * live * D + (relayer ? G * e * D : 0.0);
  const double block = T * (D + 2 * H) + e * D + n * (Dn + 4 * Dn + Dn) + (keep ? T * 3 * D + e * 2 * F : 0.0);
  const double layer = (A + 1) * T * D + e * 3 * D + A * block + (relayer ? n * Dn : 0.0);
  save += (relayer ? 1.0 : G) * layer;
  save += 2 * n * Dh + 2 * e * Dh + 2 * n + e + 2 * n;              // readout
  save += G * A * T * H + 5 * e + n * Dn + e * D + T * D + 6 * e + 30 * n;          // adjoints, edge gradients (doubles), forces, virials
  save += double(row_maxima_words(N, E)) * (relayer ? 2 : 1);       // (a layer run again takes its own)
  // tmp: the fullest scope
  const double attention_bwd = T * 5 * D + (keep ? 0.0 : T * 4 * D);
  const double norms = folds_norms() && !norms_apart_ ? 0.0 : 1.0;  // the norms' rows
  const double attention_fwd = norms * T * D + (keep ? 0.0 : T * 3 * D);
  const double edge_mlp = c * (2 * F + D) + (keep ? c * F : c * (2 * F + norms * D)) + n * 5 * Dn;  // (beside the atoms')
  const double combination = e * 4 * D + 2 * live * D;
  const double heads = 2 * n * Dh + 2 * e * Dh;
  double tmp = std::max(std::max(attention_bwd, attention_fwd), std::max(std::max(edge_mlp, combination), heads));
  tmp = std::max(tmp, n * 5 * Dn);
  need.save = size_t(save * 4.0 * 1.03) + (size_t(8) << 20);
  need.tmp = size_t(tmp * 4.0 * 1.03) + (size_t(8) << 20);
  return need;
}

// Rows whose maxima a pass keeps (class RowMaxima): what each layer, block and readout writes for a GEMM to read.
size_t Model::row_maxima_words(int N, int E) const {
  const size_t G = h_.num_gnn_layers, A = h_.num_attention_layers, T = size_t(N) + E + 64, n = size_t(N) + 64;
  if (!scales_rows(format_of(mode_))) return 0;
  return G * ((13 * A + 8) * T + 8 * A * n) + 4 * T + 6 * n;
}

size_t Model::memory_estimate(int tier, int N, int E) const {
  const MemoryNeed need = memory_need(tier, N, E, 0);
  return need.save + need.tmp;
}

int Model::choose_tier(const RunOptions& o, int N, int E) const {
  if (o.recompute != RECOMPUTE_AUTO) return o.recompute;
  for (int tier = std::max(int(RECOMPUTE_NEVER), o.tier_floor); tier < RECOMPUTE_LAYERS; ++tier)
    if (o.budget == 0 || memory_estimate(tier, N, E) <= o.budget) return tier;
  return RECOMPUTE_LAYERS;
}

PassOut Model::run_feedforward(Stream& st, Arena& save, Arena& tmp, const PackedEdges& pk, bool grad, int mode, Taps* taps,
                               const RunOptions& opt) {
  const int N = pk.N, E = pk.E, T = N + E, S = pk.M + 1;
  const int D = h_.d_pet, Dn = h_.d_node, Dh = h_.d_head, H = h_.num_heads, hd = h_.head_dim;
  const int G = h_.num_gnn_layers, A = h_.num_attention_layers;
  const Gemms gm{st, tmp};
  const float sc = float(1.0 / (std::sqrt(double(hd)) * h_.attention_temperature));
  const size_t Ea = E > 0 ? E : 1, Ta = T > 0 ? T : 1, Na = N > 0 ? N : 1;

  // taps name buffers that a recompute would overwrite or never keep: a tapped pass keeps everything
  const int tier = (taps || !grad) ? int(RECOMPUTE_NEVER) : choose_tier(opt, N, E);
  last_tier_ = tier, last_estimate_ = memory_estimate(tier, N, E);
  const bool keep_wide = tier == RECOMPUTE_NEVER, relayer = grad && tier == RECOMPUTE_LAYERS;
  const int chunk = keep_wide ? 0 : edge_chunk_rows(E);
  RowMaxima maxima(st, save, row_maxima_words(N, E) * (relayer ? 2 : 1));  // a layer run again takes its own

  struct Block {
    Rows tok, eps, node_res;  // what the block's three norms read
    float *ml, *pre_c, *pre_e;
    Rows qkv, merged;
  };
  struct Layer {
    float *cpre, *cph_pre, *out_edge;
    std::vector<Block> blk;
  };
  auto attention_args = [&](const Block& b, const Rows& qkv) {
    AttnArgs at;
    at.N = N, at.H = H, at.hd = hd, at.S = S, at.sc = sc, at.off = pk.off, at.cut = pk.cut;
    at.mode = attention_mode_for(mode), at.tf32 = wide();
    at.pairs = pk.pairs, at.T = T;
    at.qkv = qkv.p, at.merged = b.merged.p, at.ml = b.ml;
    return at;
  };
  // The RMSNorms of a block: in the GEMM that reads them, where the weight has taken the gain (Mat::after_norm), or by themselves. norm_of
  // is the input of that GEMM, normed what makes of it the GEMM of the norm, gain_of what the norm's backward multiplies by.
  const auto norm_of = [&](const Rows& x, const Mat& reader, const std::string& name, int R, int width) {
    if (reader.after_norm) return x;
    const Rows y = maxima.fresh(tmp.alloc<float>(size_t(R > 0 ? R : 1) * width), R);
    norm_fwd(st, y.p, x.p, nullptr, vec(name + ".weight"), nullptr, R, width, y.mx);
    return y;
  };
  const auto gain_of = [&](const Mat& reader, const std::string& name) { return reader.after_norm ? nullptr : vec(name + ".weight"); };
  const auto normed = [&](GemmArgs a, const Mat& reader) {
    a.rms = reader.after_norm ? 1.f : 0.f;
    return a;
  };
  const auto maxima_for = [&](const Mat& reader, size_t R) { return reader.after_norm ? maxima.take(R) : nullptr; };
  // qkv = W_in . norm(tokens) + b
  auto make_qkv = [&](const Rows& qkv, const std::string& tl, const Block& b) {
    Scope s(tmp);
    const Mat& w = mat(tl + ".attention.input_linear.weight");
    gm.one(normed(Gemms::linear_args(qkv, norm_of(b.tok, w, tl + ".norm_attention", T, D), w, vec(tl + ".attention.input_linear.bias"), T), w));
  };
  // The edge MLP's first half on rows [r0, r0 + nr): pre = W_in . norm(eps) + b and, with `he`, v * sigmoid(g).
  auto edge_mlp_in = [&](const Rows& he, float* pre, const Block& b, int r0, const std::string& tl, int nr) {
    const Mat& w = mat(tl + ".mlp.w_in.weight");
    return normed(Gemms::swiglu_args(he, pre, norm_of(b.eps.from(r0, D), w, tl + ".norm_mlp", nr, D), w, vec(tl + ".mlp.w_in.bias"), nr), w);
  };

  // One message-passing layer forward: node_in [N,Dn] -> node_out, input_edge [E,D] updated in place, saves in `sl`
  // (from `save`; the wide ones only with keep). `remote_in` [n_live, D] holds the partner rows of an exchanged list:
  // asked for from the other ranks when `ask`, else the rows a first run of this layer received.
  auto layer_forward = [&](int L, const Rows& node_in, Rows& node_out, Rows& input_edge, Layer& sl, bool keep,
                           float* remote_in, bool ask) {
    const std::string g = "gnn_layers." + std::to_string(L), ls = std::to_string(L), c0 = g + ".compress.0";
    sl.blk.resize(A);
    // Token buffers: block a's tokens are [input_node ; edge_cur]; its edge output is written
    // straight into the edge rows of block a+1's, the last one's being the layer's out_edge.
    std::vector<Rows> tokbuf(A + 1);
    for (int a = 0; a <= A; ++a) {
      tokbuf[a].p = save.alloc<float>(Ta * D);
      if (a < A) tokbuf[a].mx = maxima_for(mat(g + ".trans.layers." + std::to_string(a) + ".attention.input_linear.weight"), Ta);
    }
    sl.cpre = save.alloc<float>(Ea * D);
    const auto contraction = [&](int a, const Rows& node) {  // block a's atom tokens
      const std::string tl = g + ".trans.layers." + std::to_string(a);
      return Gemms::linear_args(tokbuf[a], node, mat(tl + ".center_contraction.weight"), vec(tl + ".center_contraction.bias"), N);
    };
    {
      Scope s0(tmp);
      const Rows cact = maxima.fresh(tmp.alloc<float>(Ea * D), Ea);
      if (L == 0) {
        compress0(st, cact.p, sl.cpre, vec(c0 + "@b"), mat(c0 + "@tab").w, mat(c0 + "@x4").w, pk, D, cact.mx);
      } else {
        gm.compress(cact, sl.cpre, input_edge, mat(c0 + "@in"), vec(c0 + "@b"), mat(c0 + "@tab"), mat(c0 + "@x4"), pk);
      }
      gm.two(contraction(0, node_in),
             Gemms::linear_args(tokbuf[0].from(N, D), cact, mat(g + ".compress.2.weight"), vec(g + ".compress.2.bias"), E));
    }
    tap(taps, "et" + ls, tokbuf[0].p + size_t(N) * D, size_t(E) * D);

    Rows node_cur = node_in;
    for (int a = 0; a < A; ++a) {
      const std::string tl = g + ".trans.layers." + std::to_string(a), tag = ls + "_" + std::to_string(a);
      Block& b = sl.blk[a];
      const Mat &w_cin = mat(tl + ".center_mlp.w_in.weight"), &w_ein = mat(tl + ".mlp.w_in.weight");
      b.tok = tokbuf[a];
      b.merged = maxima.fresh(save.alloc<float>(Ta * D), Ta);
      b.ml = save.alloc<float>(Ta * H * 2);
      b.eps = {save.alloc<float>(Ea * D), maxima_for(w_ein, Ea)};
      b.node_res = {save.alloc<float>(Na * Dn), maxima_for(w_cin, Na)};
      b.pre_c = save.alloc<float>(Na * w_cin.rows);
      b.qkv = keep ? Rows{save.alloc<float>(Ta * 3 * D)} : Rows{};
      b.pre_e = keep ? save.alloc<float>(Ea * w_ein.rows) : nullptr;
      const Rows node_next = maxima.fresh(a + 1 == A ? node_out.p : save.alloc<float>(Na * Dn), Na);
      if (a + 1 == A) node_out = node_next;
      if (a > 0) gm.one(contraction(a, node_cur));
      {
        Scope s1(tmp);
        const Rows qkv = keep ? b.qkv : Rows{tmp.alloc<float>(Ta * 3 * D)};
        make_qkv(qkv, tl, b);
        AttnArgs at = attention_args(b, qkv);
        at.merged_max = b.merged.mx;
        attention_forward(st, at);
      }
      tap(taps, "merged" + tag, b.merged.p, size_t(T) * D);
      // eps = output layer(merged) + edge_cur on the edges' rows, node_res = expansion(output layer(merged)) + node_cur on the atoms'
      gm.two(Gemms::linear_args(b.node_res, b.merged, mat(tl + "@expand"), vec(tl + "@expand_b"), N, node_cur.p, 0),
             Gemms::linear_args(b.eps, b.merged.from(N, D), mat(tl + ".attention.output_linear.weight"),
                                vec(tl + ".attention.output_linear.bias"), E, b.tok.p + size_t(N) * D, 0));
      // the atoms' MLP, and the edges' a chunk at a time: the first chunk's GEMMs share their launches with the atoms'
      Scope s2(tmp);
      const Rows hc = maxima.fresh(tmp.alloc<float>(Na * (w_cin.rows / 2)), Na);
      const Rows node_in_rows = norm_of(b.node_res, w_cin, tl + ".norm_center_features", N, Dn);
      const GemmArgs node_in_args =
          normed(Gemms::swiglu_args(hc, b.pre_c, node_in_rows, w_cin, vec(tl + ".center_mlp.w_in.bias"), N), w_cin);
      const GemmArgs node_out_args =
          Gemms::linear_args(node_next, hc, mat(tl + ".center_mlp.w_out.weight"), vec(tl + ".center_mlp.w_out.bias"), N, b.node_res.p, 0);
      const int rows = keep || chunk <= 0 ? (E > 0 ? E : 1) : chunk;
      int r0 = 0;
      do {
        const int nr = std::min(rows, E - r0);
        Scope s3(tmp);
        const Rows he = maxima.fresh(tmp.alloc<float>(size_t(nr) * (w_ein.rows / 2)), nr);
        float* pre = keep ? b.pre_e + size_t(r0) * w_ein.rows : tmp.alloc<float>(size_t(nr) * w_ein.rows);
        const GemmArgs edge_in_args = edge_mlp_in(he, pre, b, r0, tl, nr);
        const GemmArgs edge_out_args = Gemms::linear_args(tokbuf[a + 1].from(size_t(N) + r0, D), he, mat(tl + ".mlp.w_out.weight"),
                                                          vec(tl + ".mlp.w_out.bias"), nr, b.eps.p + size_t(r0) * D, 0);
        if (r0 == 0) {
          gm.two(node_in_args, edge_in_args);
          gm.two(node_out_args, edge_out_args);
        } else {
          gm.one(edge_in_args), gm.one(edge_out_args);
        }
        r0 += rows;
      } while (r0 < E);
      node_cur = node_next;
      tap(taps, "node" + tag, node_cur.p, size_t(N) * Dn);
      tap(taps, "edge" + tag, tokbuf[a + 1].p + size_t(N) * D, size_t(E) * D);
    }
    sl.out_edge = tokbuf[A].p + size_t(N) * D;
    sl.cph_pre = save.alloc<float>(Ea * 2 * D);
    {
      Scope s4(tmp);
      const Rows comb = maxima.fresh(tmp.alloc<float>(Ea * 2 * D), Ea), cph = maxima.fresh(tmp.alloc<float>(Ea * 2 * D), Ea);
      RemoteRows remote;
      if (pk.exchange) {  // edges to ghosts read their partners' rows from the ghosts' ranks (src/feedforward.cpp:171-179)
        if (ask) {
          float* send = tmp.alloc<float>(size_t(pk.n_live > 0 ? pk.n_live : 1) * D);
          gather_live(st, send, sl.out_edge, D, 0, pk.live_packed, pk.n_live, D);
          exchange_rows(st, pk, send, remote_in, D);
        }
        remote = RemoteRows{pk.remote_of, remote_in};
      }
      concat_norm_fwd(st, comb.p, sl.out_edge, pk.reverse, input_edge.p, vec("combination_norms." + ls + ".weight"),
                      vec("combination_norms." + ls + ".bias"), E, D, remote, comb.mx);
      gm.linear_silu(cph, sl.cph_pre, comb, mat("combination_mlps." + ls + ".0.weight"), vec("combination_mlps." + ls + ".0.bias"), E);
      input_edge.mx = maxima.take(Ea);
      gm.linear(input_edge, cph, mat("combination_mlps." + ls + ".2.weight"), vec("combination_mlps." + ls + ".2.bias"), E,
                input_edge.p, 0);
    }
    tap(taps, "input_edge" + ls, input_edge.p, size_t(E) * D);
  };

  // ---- forward ----
  std::vector<Layer> sav(G);
  std::vector<Rows> node_at(G + 1), ie_at(G);
  std::vector<float*> remote_in(G, nullptr);
  for (int L = 0; L <= G; ++L) node_at[L] = {save.alloc<float>(Na * Dn)};  // the nodes entering layer L; [G]: the readout's
  Rows input_edge = {save.alloc<float>(Ea * D)};  // layer 0 does not multiply it: its rows' maxima come with layer 0's output
  if (pk.exchange)
    for (int L = 0; L < G; ++L) remote_in[L] = save.alloc<float>(size_t(pk.n_live > 0 ? pk.n_live : 1) * D);
  if (relayer)
    for (int L = 0; L < G; ++L) ie_at[L] = {save.alloc<float>(Ea * D)};  // input_edge as it entered layer L
  node_at[0].mx = maxima.take(Na);
  gather_rows_two(st, node_at[0].p, mat("node_embedders.0.weight").w, pk.atom_species, N, Dn, node_at[0].mx, input_edge.p,
                  mat("edge_embedder.weight").w, pk.species, E, D);
  for (int L = 0; L < G; ++L) {
    if (relayer) {
      ie_at[L].mx = input_edge.mx;
      PETB_CUDA(cudaMemcpyAsync(ie_at[L].p, input_edge.p, sizeof(float) * size_t(E) * D, cudaMemcpyDeviceToDevice, st.s));
      Scope layer_saves(save);  // nothing of the layer is kept: the backward runs it again
      layer_forward(L, node_at[L], node_at[L + 1], input_edge, sav[L], false, remote_in[L], true);
    } else {
      layer_forward(L, node_at[L], node_at[L + 1], input_edge, sav[L], grad && keep_wide, remote_in[L], true);
    }
  }
  const Rows node = node_at[G];

  // ---- readout (src/model.cpp:656-691) ----
  float* nh0_pre = save.alloc<float>(Na * Dh);
  float* nh1_pre = save.alloc<float>(Na * Dh);
  float* eh0_pre = save.alloc<float>(Ea * Dh);
  float* eh1_pre = save.alloc<float>(Ea * Dh);
  float* node_pred = save.alloc<float>(Na);
  float* edge_pred = save.alloc<float>(Ea);
  float* net = save.alloc<float>(Na);
  double* per_atom = save.alloc<double>(pk.n_atoms > 0 ? pk.n_atoms : 1);
  {
    Scope s5(tmp);
    const Rows nh0 = maxima.fresh(tmp.alloc<float>(Na * Dh), Na), eh0 = maxima.fresh(tmp.alloc<float>(Ea * Dh), Ea);
    float* nh1 = tmp.alloc<float>(Na * Dh);
    float* eh1 = tmp.alloc<float>(Ea * Dh);
    gm.two(Gemms::silu_args(nh0, nh0_pre, node, mat("node_heads.energy.0.0.weight"), vec("node_heads.energy.0.0.bias"), N),
           Gemms::silu_args(eh0, eh0_pre, input_edge, mat("edge_heads.energy.0.0.weight"), vec("edge_heads.energy.0.0.bias"), E));
    gm.two(Gemms::silu_args({nh1}, nh1_pre, nh0, mat("node_heads.energy.0.2.weight"), vec("node_heads.energy.0.2.bias"), N),
           Gemms::silu_args({eh1}, eh1_pre, eh0, mat("edge_heads.energy.0.2.weight"), vec("edge_heads.energy.0.2.bias"), E));
    gemv_rows(st, nh1, Dh, mat("node_last_layers.energy.0.energy___0.weight").w, vec("node_last_layers.energy.0.energy___0.bias"),
              node_pred, N, Dh);
    gemv_rows(st, eh1, Dh, mat("edge_last_layers.energy.0.energy___0.weight").w, vec("edge_last_layers.energy.0.energy___0.bias"),
              edge_pred, E, Dh);
  }
  tap(taps, "node_pred", node_pred, N);
  tap(taps, "edge_pred", edge_pred, E);
  if (pk.n_atoms != N)  // (the readout writes those of the centres)
    PETB_CUDA(cudaMemsetAsync(per_atom, 0, sizeof(double) * size_t(pk.n_atoms > 0 ? pk.n_atoms : 1), st.s));
  readout_energy(st, net, per_atom, node_pred, edge_pred, pk, comp_, scale_, false, true);
  if (!grad) return finish(st, save, pk, false, nullptr, nullptr, nullptr, per_atom);

  // ---- backward (src/model.cpp:749-778, src/feedforward.cpp:199-336) ----
  float* x4_adj = save.alloc<float>(Ea * 4);
  float* cf_adj = save.alloc<float>(Ea);
  const size_t head_words = Ta * H;
  float* heads = save.alloc<float>(size_t(G) * A * head_words);  // each block's share of every head in the edges' cutoff factors,
  int blocks_done = 0;                                           // in the order of the backward
  Rows node_adj = maxima.fresh(save.alloc<float>(Na * Dn), Na), ie_adj = maxima.fresh(save.alloc<float>(Ea * D), Ea);
  Rows tok_adj = {save.alloc<float>(Ta * D)};
  {
    Scope s6(tmp);
    const Rows nh1_adj = maxima.fresh(tmp.alloc<float>(Na * Dh), Na), nh0_adj = maxima.fresh(tmp.alloc<float>(Na * Dh), Na);
    const Rows eh1_adj = maxima.fresh(tmp.alloc<float>(Ea * Dh), Ea), eh0_adj = maxima.fresh(tmp.alloc<float>(Ea * Dh), Ea);
    readout_seed_bwd(st, nh1_adj.p, mat("node_last_layers.energy.0.energy___0.weight").w, nh1_pre, nullptr, nullptr, pk.n_local, N, Dh,
                     nh1_adj.mx);
    readout_seed_bwd(st, eh1_adj.p, mat("edge_last_layers.energy.0.energy___0.weight").w, eh1_pre, pk.cut, pk.center, pk.n_local, E, Dh,
                     eh1_adj.mx);
    gm.two(Gemms::silu_bwd_args(nh0_adj, nh1_adj, mat("node_heads.energy.0.2.weight"), nh0_pre, N),
           Gemms::silu_bwd_args(eh0_adj, eh1_adj, mat("edge_heads.energy.0.2.weight"), eh0_pre, E));
    gm.two(Gemms::linear_bwd_args(node_adj, nh0_adj, mat("node_heads.energy.0.0.weight"), N, false),
           Gemms::linear_bwd_args(ie_adj, eh0_adj, mat("edge_heads.energy.0.0.weight"), E, false));
  }
  // The adjoint of a layer's tokens is one buffer written again and again: each writer of its edge rows or of all of it
  // takes fresh maxima.
  for (int L = G - 1; L >= 0; --L) {
    const std::string g = "gnn_layers." + std::to_string(L), ls = std::to_string(L), c0 = g + ".compress.0";
    Scope relayered(save);  // under Layers: this layer's saves, made again below and dropped after its backward
    Layer again;
    if (relayer) {
      Rows scratch_node = {save.alloc<float>(Na * Dn)};
      layer_forward(L, node_at[L], scratch_node, ie_at[L], again, false, remote_in[L], false);
    }
    const Layer& sl = relayer ? again : sav[L];
    {
      Scope s7(tmp);
      const Rows cph_adj = maxima.fresh(tmp.alloc<float>(Ea * 2 * D), Ea);
      float* cnorm_adj = tmp.alloc<float>(Ea * 2 * D);
      gm.linear_silu_bwd(cph_adj, ie_adj, mat("combination_mlps." + ls + ".2.weight"), sl.cph_pre, E);
      gm.linear_bwd({cnorm_adj}, cph_adj, mat("combination_mlps." + ls + ".0.weight"), E, false);
      RemoteRows remote;
      float* remote_adj = nullptr;
      if (pk.exchange) {  // the partner's rank wants the adjoint of the row this edge read (src/feedforward.cpp:241-255)
        const size_t La = size_t(pk.n_live > 0 ? pk.n_live : 1) * D;
        float* send = tmp.alloc<float>(La);
        remote_adj = tmp.alloc<float>(La);
        remote = RemoteRows{pk.remote_of, remote_in[L]};
        concat_norm_remote_bwd(st, send, cnorm_adj, sl.out_edge, vec("combination_norms." + ls + ".weight"), pk.live_packed,
                               pk.n_live, D, remote);
        exchange_rows(st, pk, send, remote_adj, D);
      }
      tok_adj.mx = maxima.take(Ta);
      const Rows edge_adj = tok_adj.from(N, D);
      concat_norm_bwd(st, edge_adj.p, cnorm_adj, sl.out_edge, pk.reverse, ie_adj.p, vec("combination_norms." + ls + ".weight"), E, D,
                      remote, remote_adj, edge_adj.mx);
    }
    for (int a = A - 1; a >= 0; --a) {
      const std::string tl = g + ".trans.layers." + std::to_string(a);
      const Block& b = sl.blk[a];
      const Mat &w_cin = mat(tl + ".center_mlp.w_in.weight"), &w_ein = mat(tl + ".mlp.w_in.weight");
      // the two MLPs: afterwards edge_adj and node_adj are eps's and node_res's
      const Rows edge_adj = tok_adj.from(N, D);  // of the MLP's output
      tok_adj.mx = maxima.take(Ta);
      const Rows eps_adj = tok_adj.from(N, D);   // the same rows once the MLP's backward has added to them
      const int rows = b.pre_e || chunk <= 0 ? (E > 0 ? E : 1) : chunk;
      {
        Scope s9(tmp);
        const Rows prec_adj = maxima.fresh(tmp.alloc<float>(Na * w_cin.rows), Na);
        float* cnorm_adj = tmp.alloc<float>(Na * Dn);
        const GemmArgs node_out_args = Gemms::swiglu_bwd_args(prec_adj, node_adj, mat(tl + ".center_mlp.w_out.weight"), b.pre_c, N);
        const GemmArgs node_in_args = Gemms::linear_bwd_args({cnorm_adj}, prec_adj, w_cin, N, false);
        int r0 = 0;
        do {
          const int nr = std::min(rows, E - r0);
          Scope s8(tmp);
          const float* eps_rows = b.eps.p + size_t(r0) * D;
          const Rows adj_rows = edge_adj.from(r0, D);
          const float* pre = b.pre_e ? b.pre_e + size_t(r0) * w_ein.rows : nullptr;
          if (!pre) {  // the pre-activation was not kept: these rows' again
            float* again_pre = tmp.alloc<float>(size_t(nr) * w_ein.rows);
            gm.one(edge_mlp_in({}, again_pre, b, r0, tl, nr));
            pre = again_pre;
          }
          const Rows pre_adj = maxima.fresh(tmp.alloc<float>(size_t(nr) * w_ein.rows), nr);
          float* enorm_adj = tmp.alloc<float>(size_t(nr) * D);
          const GemmArgs edge_out_args = Gemms::swiglu_bwd_args(pre_adj, adj_rows, mat(tl + ".mlp.w_out.weight"), pre, nr);
          const GemmArgs edge_in_args = Gemms::linear_bwd_args({enorm_adj}, pre_adj, w_ein, nr, false);
          if (r0 == 0) {
            gm.two(node_out_args, edge_out_args);
            gm.two(node_in_args, edge_in_args);
            node_adj.mx = maxima.take(Na);
            norm_bwd_two(st, node_adj.p, cnorm_adj, b.node_res.p, gain_of(w_cin, tl + ".norm_center_features"), N, Dn, node_adj.mx,
                         adj_rows.p, enorm_adj, eps_rows, gain_of(w_ein, tl + ".norm_mlp"), nr, D, eps_adj.mx);
          } else {
            gm.one(edge_out_args), gm.one(edge_in_args);
            norm_bwd_two(st, nullptr, nullptr, nullptr, nullptr, 0, Dn, nullptr, adj_rows.p, enorm_adj, eps_rows,
                         gain_of(w_ein, tl + ".norm_mlp"), nr, D, eps_adj.from(r0, D).mx);
          }
          r0 += rows;
        } while (r0 < E);
      }
      {  // attention
        Scope s10(tmp);
        const Rows dmerged = Rows{tmp.alloc<float>(Ta * D)};
        const Rows qkv_adj = maxima.fresh(tmp.alloc<float>(Ta * 3 * D), Ta);
        float* cfh = heads + size_t(blocks_done++) * head_words;
        float* attn_in_adj = tmp.alloc<float>(Ta * D);
        Rows qkv = b.qkv;
        if (!qkv.p) {
          qkv = Rows{tmp.alloc<float>(Ta * 3 * D)};
          make_qkv(qkv, tl, b);
        }
        gm.two(Gemms::linear_bwd_args(dmerged, node_adj, mat(tl + "@expand"), N, false),
               Gemms::linear_bwd_args(dmerged.from(N, D), eps_adj, mat(tl + ".attention.output_linear.weight"), E, false));
        AttnArgs at = attention_args(b, qkv);
        at.dmerged = dmerged.p, at.qkv_adj = qkv_adj.p, at.qkv_adj_max = qkv_adj.mx, at.cfh = cfh;
        attention_backward(st, at);
        const Mat& w_qkv = mat(tl + ".attention.input_linear.weight");
        gm.linear_bwd({attn_in_adj}, qkv_adj, w_qkv, T, false);
        // through the norm, back to where the tokens came from: atom rows to the contraction's
        // output adjoint (written), edge rows onto the edge residual (accumulated)
        tok_adj.mx = maxima.take(Ta);
        norm_bwd(st, tok_adj.p, attn_in_adj, b.tok.p, gain_of(w_qkv, tl + ".norm_attention"), false, T, D, N, nullptr, tok_adj.mx);
      }
      node_adj.mx = maxima.take(Na);
      gm.linear_bwd(node_adj, tok_adj, mat(tl + ".center_contraction.weight"), N, true);
    }
    {  // the edge rows are now et's
      Scope s11(tmp);
      const Rows gz = maxima.fresh(tmp.alloc<float>(Ea * D), Ea);
      gm.linear_silu_bwd(gz, tok_adj.from(N, D), mat(g + ".compress.2.weight"), sl.cpre, E);
      compress_geometry_bwd(st, x4_adj, gz.p, mat(c0 + "@x4").w, E, D, L + 1 < G);
      ie_adj.mx = maxima.take(Ea);
      if (L > 0) gm.linear_bwd(ie_adj, gz, mat(c0 + "@in"), E, true);
    }
  }
  cutoff_share(st, cf_adj, heads, head_words, blocks_done, pk.cut, N, E, H);
  tap(taps, "x4_adj", x4_adj, size_t(E) * 4);
  tap(taps, "cf_adj", cf_adj, E);
  return finish(st, save, pk, true, x4_adj, edge_pred, cf_adj, per_atom);
}

// ---- the residual featurizer ------------------------------------------------------

// Per GNN layer L: tokens = [node_embedders.L[species] ; compress(input_edge, geometry, species)];
// A PostLN blocks  tokens = LN(t + mlp(t)), t = LN(tokens + attention(tokens));  every layer is read
// out and the readouts summed; between layers input_edge = 0.5 (input_edge + out_edge of the reverse
// edge)  (src/residual.cpp:13-133 forward, :135-249 backward).
PassOut Model::run_residual(Stream& st, Arena& save, Arena& tmp, const PackedEdges& pk, bool grad, int mode, Taps* taps) {
  const int N = pk.N, E = pk.E, T = N + E, S = pk.M + 1;
  const int D = h_.d_pet, Dh = h_.d_head, H = h_.num_heads, hd = h_.head_dim;
  const int G = h_.num_gnn_layers, A = h_.num_attention_layers;
  const Gemms gm{st, tmp};
  const float sc = float(1.0 / (std::sqrt(double(hd)) * h_.attention_temperature));
  const size_t Ea = E > 0 ? E : 1, Ta = T > 0 ? T : 1, Na = N > 0 ? N : 1;
  RowMaxima maxima(st, save, row_maxima_words(N, E));

  struct Block {
    Rows qkv;
    float *merged, *ml, *s1, *s2, *pre;
  };
  struct Layer {
    float* cpre;
    float *nh0_pre, *nh1_pre, *eh0_pre, *eh1_pre, *edge_pred;
    std::vector<Block> blk;
  };
  std::vector<Layer> sav(G);

  Rows input_edge = {save.alloc<float>(Ea * D)};  // layer 0 does not multiply it
  gather_rows(st, input_edge.p, mat("edge_embedder.weight").w, pk.species, E, D);
  float* net = save.alloc<float>(Na);
  float* node_pred = save.alloc<float>(Na);
  double* per_atom = save.alloc<double>(pk.n_atoms > 0 ? pk.n_atoms : 1);
  if (pk.n_atoms != N)  // (the readout writes those of the centres)
    PETB_CUDA(cudaMemsetAsync(per_atom, 0, sizeof(double) * size_t(pk.n_atoms > 0 ? pk.n_atoms : 1), st.s));

  for (int L = 0; L < G; ++L) {
    const std::string g = "gnn_layers." + std::to_string(L), ls = std::to_string(L), c0 = g + ".compress.0";
    Layer& sl = sav[L];
    sl.blk.resize(A);
    Rows tokens = maxima.fresh(save.alloc<float>(Ta * D), Ta);
    sl.cpre = save.alloc<float>(Ea * D);
    gather_rows(st, tokens.p, mat("node_embedders." + ls + ".weight").w, pk.atom_species, N, D, tokens.mx);
    {
      Scope s0(tmp);
      const Rows cact = maxima.fresh(tmp.alloc<float>(Ea * D), Ea);
      if (L == 0) {
        compress0(st, cact.p, sl.cpre, vec(c0 + "@b"), mat(c0 + "@tab").w, mat(c0 + "@x4").w, pk, D, cact.mx);
      } else {
        gm.compress(cact, sl.cpre, input_edge, mat(c0 + "@in"), vec(c0 + "@b"), mat(c0 + "@tab"), mat(c0 + "@x4"), pk);
      }
      gm.linear(tokens.from(N, D), cact, mat(g + ".compress.2.weight"), vec(g + ".compress.2.bias"), E);
    }
    for (int a = 0; a < A; ++a) {
      const std::string tl = g + ".trans.layers." + std::to_string(a);
      Block& b = sl.blk[a];
      const Mat& w_in = mat(tl + ".mlp.w_in.weight");
      b.qkv = Rows{save.alloc<float>(Ta * 3 * D)};
      b.merged = save.alloc<float>(Ta * D);
      b.ml = save.alloc<float>(Ta * H * 2);
      b.s1 = save.alloc<float>(Ta * D);
      b.s2 = save.alloc<float>(Ta * D);
      b.pre = save.alloc<float>(Ta * w_in.rows);
      gm.linear(b.qkv, tokens, mat(tl + ".attention.input_linear.weight"), vec(tl + ".attention.input_linear.bias"), T);
      AttnArgs at;
      at.N = N, at.H = H, at.hd = hd, at.S = S, at.sc = sc, at.off = pk.off, at.cut = pk.cut;
      at.mode = attention_mode_for(mode), at.tf32 = wide();
      at.pairs = pk.pairs, at.T = T;
      const Rows merged = maxima.fresh(b.merged, Ta);
      at.qkv = b.qkv.p, at.merged = b.merged, at.ml = b.ml, at.merged_max = merged.mx;
      attention_forward(st, at);
      // s1 = attention(tokens) + tokens
      gm.linear({b.s1}, merged, mat(tl + ".attention.output_linear.weight"), vec(tl + ".attention.output_linear.bias"), T,
                tokens.p, 0);
      Scope s1(tmp);
      const Rows tok_a = maxima.fresh(tmp.alloc<float>(Ta * D), Ta), hmid = maxima.fresh(tmp.alloc<float>(Ta * w_in.rows), Ta);
      norm_fwd(st, tok_a.p, b.s1, nullptr, vec(tl + ".norm_attention.weight"), vec(tl + ".norm_attention.bias"), T, D, tok_a.mx);
      gm.linear_silu(hmid, b.pre, tok_a, w_in, vec(tl + ".mlp.w_in.bias"), T);
      // s2 = mlp(tok_a) + tok_a; tokens = LN(s2)
      gm.linear({b.s2}, hmid, mat(tl + ".mlp.w_out.weight"), vec(tl + ".mlp.w_out.bias"), T, tok_a.p, 0);
      tokens.mx = maxima.take(Ta);
      norm_fwd(st, tokens.p, b.s2, nullptr, vec(tl + ".norm_mlp.weight"), vec(tl + ".norm_mlp.bias"), T, D, tokens.mx);
    }
    tap(taps, "tokens" + ls, tokens.p, size_t(T) * D);
    // this layer's readout, summed onto the earlier layers' (src/model.cpp:656-691)
    sl.nh0_pre = save.alloc<float>(Na * Dh), sl.nh1_pre = save.alloc<float>(Na * Dh);
    sl.eh0_pre = save.alloc<float>(Ea * Dh), sl.eh1_pre = save.alloc<float>(Ea * Dh);
    sl.edge_pred = save.alloc<float>(Ea);
    {
      Scope s2(tmp);
      const Rows nh0 = maxima.fresh(tmp.alloc<float>(Na * Dh), Na), eh0 = maxima.fresh(tmp.alloc<float>(Ea * Dh), Ea);
      float* nh1 = tmp.alloc<float>(Na * Dh);
      float* eh1 = tmp.alloc<float>(Ea * Dh);
      const std::string nh = "node_heads.energy." + ls, eh = "edge_heads.energy." + ls;
      const std::string nl = "node_last_layers.energy." + ls + ".energy___0", el = "edge_last_layers.energy." + ls + ".energy___0";
      gm.two(Gemms::silu_args(nh0, sl.nh0_pre, tokens, mat(nh + ".0.weight"), vec(nh + ".0.bias"), N),
             Gemms::silu_args(eh0, sl.eh0_pre, tokens.from(N, D), mat(eh + ".0.weight"), vec(eh + ".0.bias"), E));
      gm.two(Gemms::silu_args({nh1}, sl.nh1_pre, nh0, mat(nh + ".2.weight"), vec(nh + ".2.bias"), N),
             Gemms::silu_args({eh1}, sl.eh1_pre, eh0, mat(eh + ".2.weight"), vec(eh + ".2.bias"), E));
      gemv_rows(st, nh1, Dh, mat(nl + ".weight").w, vec(nl + ".bias"), node_pred, N, Dh);
      gemv_rows(st, eh1, Dh, mat(el + ".weight").w, vec(el + ".bias"), sl.edge_pred, E, Dh);
      readout_energy(st, net, per_atom, node_pred, sl.edge_pred, pk, comp_, scale_, L > 0, L + 1 == G);
      tap(taps, "node_pred" + ls, node_pred, N);
      tap(taps, "edge_pred" + ls, sl.edge_pred, E);
      tap(taps, "net" + ls, net, N);
    }
    if (L + 1 < G) {
      RemoteRows remote;
      if (pk.exchange) {  // src/residual.cpp:123-132
        const size_t La = size_t(pk.n_live > 0 ? pk.n_live : 1) * D;
        float* send = tmp.alloc<float>(La);
        float* recv = tmp.alloc<float>(La);
        gather_live(st, send, tokens.p + size_t(N) * D, D, 0, pk.live_packed, pk.n_live, D);
        exchange_rows(st, pk, send, recv, D);
        remote = RemoteRows{pk.remote_of, recv};
      }
      input_edge.mx = maxima.take(Ea);
      message_average(st, input_edge.p, tokens.p + size_t(N) * D, pk.reverse, E, D, remote, input_edge.mx);
    }
  }
  if (!grad) return finish(st, save, pk, false, nullptr, nullptr, nullptr, per_atom);

  // ---- backward ----
  float* x4_adj = save.alloc<float>(Ea * 4);
  float* cf_adj = save.alloc<float>(Ea);
  float* cutoff_adj = save.alloc<float>(Ea);  // sum over layers of the edge predictions
  const size_t head_words = Ta * H;
  float* heads = save.alloc<float>(size_t(G) * A * head_words);  // each block's share of every head in the edges' cutoff factors,
  int blocks_done = 0;                                           // in the order of the backward
  PETB_CUDA(cudaMemcpyAsync(cutoff_adj, sav[0].edge_pred, sizeof(float) * Ea, cudaMemcpyDeviceToDevice, st.s));
  for (int L = 1; L < G; ++L) add_inplace(st, cutoff_adj, sav[L].edge_pred, size_t(E));
  float* ie_a = save.alloc<float>(Ea * D);
  float* ie_b = save.alloc<float>(Ea * D);
  float* ie_adj = ie_a;  // adjoint of the next layer's input_edge
  for (int L = G - 1; L >= 0; --L) {
    const std::string g = "gnn_layers." + std::to_string(L), ls = std::to_string(L), c0 = g + ".compress.0";
    const Layer& sl = sav[L];
    Scope layer_scope(tmp);
    Rows tokens_adj = {tmp.alloc<float>(Ta * D)};
    float* alt = tmp.alloc<float>(Ta * D);
    {  // the readout's adjoint of this layer's tokens
      Scope s3(tmp);
      const Rows nh1_adj = maxima.fresh(tmp.alloc<float>(Na * Dh), Na), nh0_adj = maxima.fresh(tmp.alloc<float>(Na * Dh), Na);
      const Rows eh1_adj = maxima.fresh(tmp.alloc<float>(Ea * Dh), Ea), eh0_adj = maxima.fresh(tmp.alloc<float>(Ea * Dh), Ea);
      const std::string nh = "node_heads.energy." + ls, eh = "edge_heads.energy." + ls;
      const std::string nl = "node_last_layers.energy." + ls + ".energy___0", el = "edge_last_layers.energy." + ls + ".energy___0";
      readout_seed_bwd(st, nh1_adj.p, mat(nl + ".weight").w, sl.nh1_pre, nullptr, nullptr, pk.n_local, N, Dh, nh1_adj.mx);
      readout_seed_bwd(st, eh1_adj.p, mat(el + ".weight").w, sl.eh1_pre, pk.cut, pk.center, pk.n_local, E, Dh, eh1_adj.mx);
      gm.two(Gemms::silu_bwd_args(nh0_adj, nh1_adj, mat(nh + ".2.weight"), sl.nh0_pre, N),
             Gemms::silu_bwd_args(eh0_adj, eh1_adj, mat(eh + ".2.weight"), sl.eh0_pre, E));
      gm.two(Gemms::linear_bwd_args(tokens_adj, nh0_adj, mat(nh + ".0.weight"), N, false),
             Gemms::linear_bwd_args(tokens_adj.from(N, D), eh0_adj, mat(eh + ".0.weight"), E, false));
    }
    float* ie_next = ie_adj == ie_a ? ie_b : ie_a;
    if (L + 1 < G) {
      RemoteRows remote;
      if (pk.exchange) {  // src/residual.cpp:189
        const size_t La = size_t(pk.n_live > 0 ? pk.n_live : 1) * D;
        float* send = tmp.alloc<float>(La);
        float* recv = tmp.alloc<float>(La);
        gather_live(st, send, ie_adj, D, 0, pk.live_packed, pk.n_live, D);
        exchange_rows(st, pk, send, recv, D);
        remote = RemoteRows{pk.remote_of, recv};
      }
      message_average_bwd(st, ie_next, tokens_adj.p + size_t(N) * D, ie_adj, pk.reverse, E, D, remote);
    }
    else PETB_CUDA(cudaMemsetAsync(ie_next, 0, sizeof(float) * Ea * D, st.s));
    for (int a = A - 1; a >= 0; --a) {
      const std::string tl = g + ".trans.layers." + std::to_string(a);
      const Block& b = sl.blk[a];
      const Mat& w_in = mat(tl + ".mlp.w_in.weight");
      Scope s4(tmp);
      const Rows s2_adj = maxima.fresh(tmp.alloc<float>(Ta * D), Ta);
      float* tok_a_adj = tmp.alloc<float>(Ta * D);
      // tokens_out = LN(s2), s2 = tok_a + mlp(tok_a)
      norm_bwd(st, s2_adj.p, tokens_adj.p, b.s2, vec(tl + ".norm_mlp.weight"), true, T, D, T, tok_a_adj, s2_adj.mx);
      {
        Scope s5(tmp);
        const Rows h_adj = maxima.fresh(tmp.alloc<float>(Ta * w_in.rows), Ta);
        gm.linear_silu_bwd(h_adj, s2_adj, mat(tl + ".mlp.w_out.weight"), b.pre, T);
        gm.linear_bwd({tok_a_adj}, h_adj, w_in, T, true);
      }
      // tok_a = LN(s1), s1 = tokens_in + attention(tokens_in)
      Rows s1_adj = maxima.fresh(alt, Ta);
      norm_bwd(st, s1_adj.p, tok_a_adj, b.s1, vec(tl + ".norm_attention.weight"), true, T, D, T, nullptr, s1_adj.mx);
      {
        Scope s6(tmp);
        const Rows dmerged = Rows{tmp.alloc<float>(Ta * D)};
        const Rows qkv_adj = maxima.fresh(tmp.alloc<float>(Ta * 3 * D), Ta);
        float* cfh = heads + size_t(blocks_done++) * head_words;
        gm.linear_bwd(dmerged, s1_adj, mat(tl + ".attention.output_linear.weight"), T, false);
        AttnArgs at;
        at.N = N, at.H = H, at.hd = hd, at.S = S, at.sc = sc, at.off = pk.off, at.cut = pk.cut;
      at.mode = attention_mode_for(mode), at.tf32 = wide();
        at.pairs = pk.pairs, at.T = T;
        at.qkv = b.qkv.p, at.merged = b.merged, at.ml = b.ml, at.dmerged = dmerged.p;
        at.qkv_adj = qkv_adj.p, at.cfh = cfh;
        at.qkv_adj_max = qkv_adj.mx;
        attention_backward(st, at);
        s1_adj.mx = maxima.take(Ta);
        gm.linear_bwd(s1_adj, qkv_adj, mat(tl + ".attention.input_linear.weight"), T, true);
      }
      alt = tokens_adj.p;
      tokens_adj = s1_adj;
    }
    {  // tokens = [node_L ; et]: only et depends on the geometry
      Scope s7(tmp);
      const Rows gz = maxima.fresh(tmp.alloc<float>(Ea * D), Ea);
      gm.linear_silu_bwd(gz, tokens_adj.from(N, D), mat(g + ".compress.2.weight"), sl.cpre, E);
      compress_geometry_bwd(st, x4_adj, gz.p, mat(c0 + "@x4").w, E, D, L + 1 < G);
      if (L > 0) gm.linear_bwd({ie_next}, gz, mat(c0 + "@in"), E, true);
    }
    ie_adj = ie_next;
  }
  cutoff_share(st, cf_adj, heads, head_words, blocks_done, pk.cut, N, E, H);
  return finish(st, save, pk, true, x4_adj, cutoff_adj, cf_adj, per_atom);
}

}  // namespace petb
