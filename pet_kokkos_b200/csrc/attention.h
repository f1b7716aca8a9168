// Per-atom multi-head attention over neighbour tokens: see attention.cu.
#pragma once

#include "common.h"

namespace petb {

enum AttnMode { ATTN_NATIVE = 0, ATTN_TF32X3 = 1, ATTN_TF32 = 2 };

struct AttnArgs {
  int N = 0, H = 0, hd = 0, S = 0;  // atoms, heads, head_dim, most tokens of any atom (max neighbours + 1)
  float sc = 1.f;                   // 1 / (sqrt(head_dim) * temperature)
  // How the products run (the reference's AttentionMode, include/pet/gemm.hpp): ATTN_NATIVE, operands in three fp16 parts (fp32
  // accuracy); ATTN_TF32X3, in two, as accurate but for the tensor core's truncating accumulate; ATTN_TF32, in one of eleven
  // bits (a speed mode, about three decimal digits). On the CUDA cores in fp32 where no tensor-core kernel takes the shape.
  int mode = 0;
  bool tf32 = false;                // forward: the tensor-core modes on tf32 instructions (where energies depend on their bits)
  double pairs = 0.0;               // sum over atoms of tokens^2 (work accounting only)
  double T = 0.0;                   // token rows (work accounting only)
  const int* off = nullptr;         // [N+1] each atom's range of edge rows
  const float* cut = nullptr;       // [E] cutoff factor of each edge token
  const float* qkv = nullptr;       // [T,3D] columns Q | K | V
  float* merged = nullptr;          // [T,D] attention output before the output projection
  uint32_t* merged_max = nullptr;   // [T] unless null, each row's largest |merged| is raised into it (zeroed by the caller)
  float* ml = nullptr;              // [T,H,2] each query's running max and 1/sum (null: not saved)
  // backward
  const float* dmerged = nullptr;   // [T,D]
  float* qkv_adj = nullptr;         // [T,3D]
  uint32_t* qkv_adj_max = nullptr;  // [T] unless null, each row's largest |qkv_adj| likewise
  float* cfh = nullptr;             // [T,H] each key's score adjoint summed over its queries
};

void attention_forward(Stream& st, const AttnArgs& a);
void attention_backward(Stream& st, const AttnArgs& a);

}  // namespace petb
