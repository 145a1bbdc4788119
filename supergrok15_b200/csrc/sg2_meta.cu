// Meta-network bookkeeping of SuperGrok v2 in single launches (sm_100a): the packed weight vector with its folded affine tables, the chain
// rule from the tables back to the meta-network's parameters, and the unit validation gradients of a bilevel step.  Each of these was a
// chain of 60 to 400 element-sized PyTorch calls: a bilevel step of the 422,755-parameter race model spent 15 ms on 1,337 launches
// with 8 ms of work on the device.
#include "sg_native.h"
#include "sg2_meta.h"
#include "optim_math.cuh"

namespace sg {
namespace {
using P = SG2Pack;

struct Seg { const float* src; int dst, n, cols; };           // cols > 0: rows of `cols` values, zero-padded to 16
struct PackArgs { Seg s[SG2_META_TENSORS]; float* out; };

// x_t, z_t, dt_t, b_t, c_t [16][3] of one direction in fp64 (see ops/sg2.py: every scan input is affine in (g, s)); `w` holds the raw
// weights of the packed vector's layout.  xz: [32][3] (x, z); rest [3][16][3] (dt, B, C).  All threads of the block.
__device__ void fold(const float* __restrict__ in_w, const float* __restrict__ in_b, const float* __restrict__ in_proj, const float* __restrict__ dtw,
                     const float* __restrict__ dtb, const float* __restrict__ bw, const float* __restrict__ cw, double* xz, double* rest) {
    for (int i = threadIdx.x; i < 96; i += blockDim.x) {
        const int r = i / 3, k = i % 3;
        double a = 0.0;
        for (int d = 0; d < 8; ++d) a += (double)in_proj[r * 8 + d] * (k < 2 ? (double)in_w[d * 2 + k] : (double)in_b[d]);
        xz[i] = a;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 144; i += blockDim.x) {
        const int m = i / 48, r = (i % 48) / 3, k = i % 3;
        const float* W = (m == 0 ? dtw : m == 1 ? bw : cw) + r * 16;
        double a = 0.0;
        for (int q = 0; q < 16; ++q) a += (double)W[q] * xz[q * 3 + k];
        if (m == 0 && k == 2) a += (double)dtb[r];
        rest[i] = a;
    }
    __syncthreads();
}

// CTA b < SG2_META_TENSORS copies tensor b to its place; two more fold the tables of a direction.
__global__ void __launch_bounds__(256) sg2_pack_kernel(const __grid_constant__ PackArgs a) {
    const int b = blockIdx.x;
    if (b < SG2_META_TENSORS) {
        const Seg s = a.s[b];
        if (s.cols == 0) for (int i = threadIdx.x; i < s.n; i += 256) a.out[s.dst + i] = s.src[i];
        else for (int i = threadIdx.x; i < s.n; i += 256) a.out[s.dst + i] = (i & 15) < s.cols ? s.src[(i >> 4) * s.cols + (i & 15)] : 0.f;
        return;
    }
    __shared__ double xz[96], rest[144];
    const int dir = b - SG2_META_TENSORS;
    const Seg* d = a.s + 2 + 9 * dir;                          // in_proj, dt weight, dt bias, B, C, ...
    fold(a.s[0].src, a.s[1].src, d[0].src, d[1].src, d[2].src, d[3].src, d[4].src, xz, rest);
    float* o = a.out + (dir == 0 ? P::AFF0 : P::AFF1);
    for (int i = threadIdx.x; i < 48; i += 256) { o[P::A_X + i] = (float)xz[i]; o[P::A_Z + i] = (float)xz[48 + i]; }
    for (int i = threadIdx.x; i < 144; i += 256) o[P::A_DT + i] = (float)rest[i];          // A_DT, A_B, A_C follow one another
}

// Gradients of the scan's own parameters and of the folded tables ([2][ng], layout in sg2_bilevel.cuh) -> gradients of input_proj and of
// both directions' parameters, in the packed vector's layout (the first GRU_WZ floats).  One CTA, fp64, fixed order.
__global__ void __launch_bounds__(256) sg2_fold_bwd_kernel(const float* __restrict__ w, const float* __restrict__ grads, int ng, float* __restrict__ out) {
    __shared__ double xz[96], rest[144], dxz[96], dinp[2][24];
    for (int dir = 0; dir < 2; ++dir) {
        const float* W = w + (dir == 0 ? P::DIR0 : P::DIR1);
        const float* G = grads + dir * ng;
        const float *dX = G + 400, *dZ = G + 448, *dR = G + 496;                 // dR: dt, B, C tables, 48 values each
        float* o = out + (dir == 0 ? P::DIR0 : P::DIR1);
        fold(w + P::IN_W, w + P::IN_B, W + P::D_INPROJ, W + P::D_DTW, W + P::D_DTB, W + P::D_BW, W + P::D_CW, xz, rest);
        for (int i = threadIdx.x; i < 96; i += 256) {
            const int r = i / 3, k = i % 3;
            double a;
            if (r < 16) {                                                        // x feeds dt, B and C
                a = (double)dX[i];
                for (int q = 0; q < 16; ++q)
                    a += (double)W[P::D_DTW + q * 16 + r] * dR[q * 3 + k] + (double)W[P::D_BW + q * 16 + r] * dR[48 + q * 3 + k] +
                         (double)W[P::D_CW + q * 16 + r] * dR[96 + q * 3 + k];
            } else a = (double)dZ[i - 48];
            dxz[i] = a;
        }
        for (int i = threadIdx.x; i < 768; i += 256) {                            // dt / B / C weights: table gradient . x^T
            const int m = i / 256, r = (i % 256) / 16, q = i % 16;
            double a = 0.0;
            for (int k = 0; k < 3; ++k) a += (double)dR[48 * m + r * 3 + k] * xz[q * 3 + k];
            o[(m == 0 ? P::D_DTW : m == 1 ? P::D_BW : P::D_CW) + i % 256] = (float)a;
        }
        for (int i = threadIdx.x; i < 16; i += 256) o[P::D_DTB + i] = dR[i * 3 + 2];
        for (int i = threadIdx.x; i < 256; i += 256) o[P::D_ALOG + i] = G[i];
        for (int i = threadIdx.x; i < 128; i += 256) { o[P::D_ROPE + i] = G[256 + i]; o[P::D_OUT + i] = G[640 + i]; }
        for (int i = threadIdx.x; i < 16; i += 256) o[P::D_D + i] = G[384 + i];
        __syncthreads();
        for (int i = threadIdx.x; i < 256; i += 256) {                            // in_proj [32][8]: d(xz) . inp^T
            const int r = i / 8, d = i % 8;
            o[P::D_INPROJ + i] = (float)(dxz[r * 3] * (double)w[P::IN_W + 2 * d] + dxz[r * 3 + 1] * (double)w[P::IN_W + 2 * d + 1] +
                                         dxz[r * 3 + 2] * (double)w[P::IN_B + d]);
        }
        for (int i = threadIdx.x; i < 24; i += 256) {
            const int d = i / 3, k = i % 3;
            double a = 0.0;
            for (int r = 0; r < 32; ++r) a += (double)W[P::D_INPROJ + r * 8 + d] * dxz[r * 3 + k];
            dinp[dir][i] = a;
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < 24; i += 256) {
        const int d = i / 3, k = i % 3;
        const float v = (float)(dinp[0][i] + dinp[1][i]);
        if (k < 2) out[P::IN_W + 2 * d + k] = v; else out[P::IN_B + d] = v;
    }
}

__device__ __forceinline__ int unit_locate(const MTArgs& a, int64_t& begin, int64_t& end) {
    int lo = 0, hi = a.n;
    const int b = blockIdx.x;
    while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (a.blk_start[mid] <= b) lo = mid; else hi = mid; }
    begin = (int64_t)(b - a.blk_start[lo]) * MT_CHUNK;
    const int64_t n = a.numel[lo];
    end = begin + MT_CHUNK < n ? begin + MT_CHUNK : n;
    return lo;
}

// per CTA: sum of squares of the finite entries, number of the others
template <typename T>
__global__ void __launch_bounds__(MT_THREADS) sg2_unit_norm_kernel(const __grid_constant__ MTArgs a, float* __restrict__ partials) {
    __shared__ float red[32];
    int64_t begin, end;
    const int t = unit_locate(a, begin, end);
    const T* g = reinterpret_cast<const T*>(a.ptr[1][t]);
    float sq = 0.f, bad = 0.f;
    for (int64_t i = begin + threadIdx.x; i < end; i += MT_THREADS) {
        const float v = Cvt<T>::to(g[i]);
        if (isfinite(v)) sq = fmaf(v, v, sq); else bad += 1.f;
    }
    sq = block_sum(sq, red);
    bad = block_sum(bad, red);
    if (threadIdx.x == 0) { float* o = partials + 3 * (int64_t)(a.blk_off + blockIdx.x); o[0] = sq; o[1] = bad; o[2] = 0.f; }
}

// out[off + i] = g[i] / |g|; a tensor with a non-finite entry contributes zeros, one without length its own values
template <typename T>
__global__ void __launch_bounds__(MT_THREADS) sg2_unit_write_kernel(const __grid_constant__ MTArgs a, const float* __restrict__ totals, float* __restrict__ out) {
    int64_t begin, end;
    const int t = unit_locate(a, begin, end);
    const T* g = reinterpret_cast<const T*>(a.ptr[1][t]);
    const int64_t off = (int64_t)reinterpret_cast<intptr_t>(a.ptr[6][t]);
    const float norm = sqrtf(totals[3 * (a.t_off + t)]);
    const bool ok = totals[3 * (a.t_off + t) + 1] == 0.f;
    const float scale = norm > 1e-12f ? 1.f / norm : 1.f;
    for (int64_t i = begin + threadIdx.x; i < end; i += MT_THREADS) out[off + i] = ok ? Cvt<T>::to(g[i]) * scale : 0.f;
}

}  // namespace

void sg2_pack(const float* const* src, int expert_hidden, float* out, cudaStream_t s) {
    PackArgs a{};
    int k = 0;
    const auto put = [&](int dst, int n, int cols = 0) { a.s[k] = Seg{src[k], dst, n, cols}; ++k; };
    put(P::IN_W, 16); put(P::IN_B, 8);
    for (int dir = 0; dir < 2; ++dir) {
        const int b = dir == 0 ? P::DIR0 : P::DIR1;
        put(b + P::D_INPROJ, 256); put(b + P::D_DTW, 256); put(b + P::D_DTB, 16); put(b + P::D_BW, 256); put(b + P::D_CW, 256);
        put(b + P::D_ALOG, 256); put(b + P::D_D, 16); put(b + P::D_ROPE, 128); put(b + P::D_OUT, 128);
    }
    put(P::GRU_WZ, 88); put(P::GRU_WR, 88); put(P::GRU_WH, 88); put(P::GRU_BZ, 4); put(P::GRU_BR, 4); put(P::GRU_BH, 4);
    for (int h = 0; h < SG2_HEADS; ++h) put(P::PQ + 176 * h, 176);
    for (int h = 0; h < SG2_HEADS; ++h) put(P::KA + 48 * h, 48);
    for (int h = 0; h < SG2_HEADS; ++h) put(P::KB + 48 * h, 48);
    put(P::EW1, SG2_NE * SG2_EH, expert_hidden); put(P::EB1, SG2_NE * SG2_EH, expert_hidden); put(P::EW2, SG2_NE * SG2_EH, expert_hidden);
    put(P::EB2, SG2_NE);
    static_assert(SG2_META_TENSORS == 2 + 18 + 6 + 12 + 4, "tensors of the meta-network");
    a.out = out;
    count_launch();
    sg2_pack_kernel<<<SG2_META_TENSORS + 2, 256, 0, s>>>(a);
}

// element counts the caller has to check: the k-th source tensor of sg2_pack
int sg2_pack_numel(int k, int expert_hidden) {
    static const int dir[9] = {256, 256, 16, 256, 256, 256, 16, 128, 128};
    if (k < 2) return k == 0 ? 16 : 8;
    if (k < 20) return dir[(k - 2) % 9];
    if (k < 23) return 88;
    if (k < 26) return 4;
    if (k < 30) return 176;
    if (k < 38) return 48;
    return k < 41 ? SG2_NE * expert_hidden : SG2_NE;
}

void sg2_fold_bwd(const float* packed, const float* grads, int ng, float* out, cudaStream_t s) {
    count_launch();
    sg2_fold_bwd_kernel<<<1, 256, 0, s>>>(packed, grads, ng, out);
}

void sg2_unit_norm(int dtype, const MTArgs& a, float* partials, cudaStream_t s) {
    const int blocks = a.blk_start[a.n];
    if (blocks <= 0) return;
    count_launch();
    switch (dtype) {
        case F32:  sg2_unit_norm_kernel<float><<<blocks, MT_THREADS, 0, s>>>(a, partials); break;
        case BF16: sg2_unit_norm_kernel<__nv_bfloat16><<<blocks, MT_THREADS, 0, s>>>(a, partials); break;
        default:   sg2_unit_norm_kernel<__half><<<blocks, MT_THREADS, 0, s>>>(a, partials); break;
    }
}

void sg2_unit_write(int dtype, const MTArgs& a, const float* totals, float* out, cudaStream_t s) {
    const int blocks = a.blk_start[a.n];
    if (blocks <= 0) return;
    count_launch();
    switch (dtype) {
        case F32:  sg2_unit_write_kernel<float><<<blocks, MT_THREADS, 0, s>>>(a, totals, out); break;
        case BF16: sg2_unit_write_kernel<__nv_bfloat16><<<blocks, MT_THREADS, 0, s>>>(a, totals, out); break;
        default:   sg2_unit_write_kernel<__half><<<blocks, MT_THREADS, 0, s>>>(a, totals, out); break;
    }
}

}  // namespace sg
