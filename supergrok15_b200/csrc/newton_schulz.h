// Newton-Schulz iteration over groups of equal-shaped matrices (newton_schulz.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime_api.h>

namespace sg {

// `batch` matrices [r, c], stored one after the other.  Row pitches: bf16 buffers are padded to 8 elements, out32 to 4.
struct NsGroup {
    int r, c, batch;
    __nv_bfloat16* x0;          // [batch, r, c] in: the normalised matrices
    __nv_bfloat16* x1;          // [batch, r, c] scratch (iterates alternate between x0 and x1)
    __nv_bfloat16* g;           // [batch, n, n] scratch, n = min(r, c)
    __nv_bfloat16* p;           // [batch, n, n] scratch
    float* out32;               // [batch, r, c] out
};

// dst[t] (bf16 rows padded to 8) = src[t] (dense fp32 [rows, cols]) * inv[t]; inv may be null
void ns_cast(const float* const* src, void* const* dst, const int* rows, const int* cols, int n, const float* inv, cudaStream_t s);
// `steps` iterations of X <- aX + b(XX^T)X + c(XX^T)^2 X on every matrix of every group; 0 on success.  `err` (device int) becomes
// non-zero when a pipeline wait ran out.
int ns_iterate(const NsGroup* groups, int n, int steps, float a, float b, float c, int* err, cudaStream_t s);

// the tile order of the symmetric products, for host-side checks
int ns_sym_tile_count(int n, int bn);
void ns_sym_tile_coords(int tile, int bn, int* m0, int* n0, int* mirror);

}  // namespace sg
