// Launchers of sg2_meta.cu.
#pragma once
#include "sg_native.h"

namespace sg {
// input_proj (2), nine tensors per direction, GRU (6), queries and both sub-key sets of four heads (12), experts (4), in the order of
// the packed vector
constexpr int SG2_META_TENSORS = 42;
int sg2_pack_numel(int k, int expert_hidden);
void sg2_pack(const float* const* src, int expert_hidden, float* out, cudaStream_t s);
void sg2_fold_bwd(const float* packed, const float* grads, int ng, float* out, cudaStream_t s);
void sg2_unit_norm(int dtype, const MTArgs& a, float* partials, cudaStream_t s);
void sg2_unit_write(int dtype, const MTArgs& a, const float* totals, float* out, cudaStream_t s);
}  // namespace sg
