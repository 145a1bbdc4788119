// Model-side kernels for the small-sequence transformers of the grokking tasks (sm_100a):
//   * causal multi-head attention for very short sequences (S <= 8) - a group of lanes per (batch, head), the whole
//     S x S score matrix lives in registers; forward and backward (scores recomputed, nothing saved but q,k,v);
//   * LayerNorm with fused residual add, forward and backward (deterministic two-stage column reduction for
//     the weight / bias gradients, no atomics).
// They replace nn.MultiheadAttention / nn.LayerNorm of the reference model (grokking_race_v2.py:310-331); library
// flash-attention kernels are tuned for long sequences and take ~2.5 ms per layer on a [8192, 8, 4, 64] problem
// whose memory traffic is worth ~20 us.
#include "sg_native.h"
#include "optim_math.cuh"

namespace sg {
namespace {

// EPL consecutive head-dim elements owned by one lane, held as loaded (packed) until they are used.  VEC: one access of EPL elements,
// which has to be aligned to its size; otherwise element by element.
template <typename T, int EPL, bool VEC> struct LaneVec {
    static constexpr int W = (EPL * (int)sizeof(T) + 3) / 4;           // 32-bit words (one half-filled for a single 16-bit element)
    static_assert(!VEC || W == 2 || W == 4, "accesses of 8 or 16 bytes");
    uint32_t w[W];
    __device__ __forceinline__ void ld(const T* p) {
        if constexpr (!VEC && sizeof(T) == 4) {
#pragma unroll
            for (int e = 0; e < EPL; ++e) w[e] = reinterpret_cast<const uint32_t*>(p)[e];
        } else if constexpr (!VEC) {
            const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
#pragma unroll
            for (int k = 0; k < W; ++k) w[k] = h[2 * k] | (2 * k + 1 < EPL ? (uint32_t)h[2 * k + 1] << 16 : 0u);
        } else if constexpr (W == 4) { const uint4 t = *reinterpret_cast<const uint4*>(p); w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w; }
        else { const uint2 t = *reinterpret_cast<const uint2*>(p); w[0] = t.x; w[1] = t.y; }
    }
    __device__ __forceinline__ float get(int e) const {
        if constexpr (sizeof(T) == 4) return __uint_as_float(w[e]);
        else return __uint_as_float((e & 1) ? (w[e >> 1] & 0xffff0000u) : (w[e >> 1] << 16));      // bf16 is the upper half of an fp32
    }
    static __device__ __forceinline__ void st(T* p, const float (&v)[EPL]) {
        T h[EPL];
#pragma unroll
        for (int e = 0; e < EPL; ++e) h[e] = Cvt<T>::from(v[e]);
        if constexpr (!VEC) {
#pragma unroll
            for (int e = 0; e < EPL; ++e) p[e] = h[e];
        } else if constexpr (W == 4) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(h);
        else *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
    }
};
// sum over the LG lanes (aligned group) of one head; every lane gets the result
template <int LG> __device__ __forceinline__ float group_sum(float x) {
#pragma unroll
    for (int o = LG / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// qkv [B, S, 3, H, HD], out [B, S, H, HD]; scale = 1/sqrt(HD).  HD / EPL lanes per (b, h): with sixteen bytes per lane a warp holds four heads
// of 64 bf16, a load instruction moves 512 bytes and one shuffle step of a score serves all four (a warp per head loaded four bytes per
// lane and spent 50 shuffles on ten scores: 37 us forward and 64 us backward for [8192, 4, 3 x 512] bf16, 134 and 235 MB).
template <typename T, int S, int EPL, int HD, bool CAUSAL, bool VEC>
__global__ void __launch_bounds__(128) attn_small_fwd_kernel(const T* __restrict__ qkv, T* __restrict__ out, int B, int H, float scale) {
    constexpr int LG = HD / EPL, PER_CTA = 128 / LG;
    const int64_t w0 = (int64_t)blockIdx.x * PER_CTA + threadIdx.x / LG;
    const bool live = w0 < (int64_t)B * H;                // idle groups run along on head 0: the shuffles take whole warps
    const int64_t w = live ? w0 : 0;
    const int b = (int)(w / H), h = (int)(w % H), l = threadIdx.x % LG;
    const int64_t D = (int64_t)H * HD;
    LaneVec<T, EPL, VEC> q[S], k[S], v[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const T* base = qkv + ((int64_t)b * S + s) * 3 * D + (int64_t)h * HD + l * EPL;
        q[s].ld(base); k[s].ld(base + D); v[s].ld(base + 2 * D);
    }
    float sc[S][S];
#pragma unroll
    for (int i = 0; i < S; ++i)
#pragma unroll
        for (int j = 0; j < S; ++j) {
            if (CAUSAL && j > i) { sc[i][j] = 0.f; continue; }
            float d = 0.f;
#pragma unroll
            for (int e = 0; e < EPL; ++e) d = fmaf(q[i].get(e), k[j].get(e), d);
            sc[i][j] = group_sum<LG>(d) * scale;
        }
#pragma unroll
    for (int i = 0; i < S; ++i) {
        const int jm = CAUSAL ? i : S - 1;
        float mx = sc[i][0];
#pragma unroll
        for (int j = 1; j < S; ++j) if (j <= jm) mx = fmaxf(mx, sc[i][j]);
        float den = 0.f;
#pragma unroll
        for (int j = 0; j < S; ++j) if (j <= jm) { sc[i][j] = __expf(sc[i][j] - mx); den += sc[i][j]; }
        const float inv = 1.f / den;
        float o[EPL];
#pragma unroll
        for (int e = 0; e < EPL; ++e) o[e] = 0.f;
#pragma unroll
        for (int j = 0; j < S; ++j) if (j <= jm) {
#pragma unroll
            for (int e = 0; e < EPL; ++e) o[e] = fmaf(sc[i][j] * inv, v[j].get(e), o[e]);
        }
        if (live) LaneVec<T, EPL, VEC>::st(out + ((int64_t)b * S + i) * D + (int64_t)h * HD + l * EPL, o);
    }
}

template <typename T, int S, int EPL, int HD, bool CAUSAL, bool VEC>
__global__ void __launch_bounds__(128) attn_small_bwd_kernel(const T* __restrict__ qkv, const T* __restrict__ dout, T* __restrict__ dqkv,
                                                             int B, int H, float scale) {
    constexpr int LG = HD / EPL, PER_CTA = 128 / LG;
    const int64_t w0 = (int64_t)blockIdx.x * PER_CTA + threadIdx.x / LG;
    const bool live = w0 < (int64_t)B * H;
    const int64_t w = live ? w0 : 0;
    const int b = (int)(w / H), h = (int)(w % H), l = threadIdx.x % LG;
    const int64_t D = (int64_t)H * HD;
    LaneVec<T, EPL, VEC> q[S], k[S], v[S], dO[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const T* base = qkv + ((int64_t)b * S + s) * 3 * D + (int64_t)h * HD + l * EPL;
        q[s].ld(base); k[s].ld(base + D); v[s].ld(base + 2 * D);
        dO[s].ld(dout + ((int64_t)b * S + s) * D + (int64_t)h * HD + l * EPL);
    }
    float p[S][S], dp[S][S];
#pragma unroll
    for (int i = 0; i < S; ++i)
#pragma unroll
        for (int j = 0; j < S; ++j) {
            if (CAUSAL && j > i) { p[i][j] = 0.f; dp[i][j] = 0.f; continue; }
            float d = 0.f, e2 = 0.f;
#pragma unroll
            for (int e = 0; e < EPL; ++e) { d = fmaf(q[i].get(e), k[j].get(e), d); e2 = fmaf(dO[i].get(e), v[j].get(e), e2); }
            p[i][j] = group_sum<LG>(d) * scale;
            dp[i][j] = group_sum<LG>(e2);
        }
#pragma unroll
    for (int i = 0; i < S; ++i) {                            // p -> probabilities, dp -> gradient of the scaled scores
        const int jm = CAUSAL ? i : S - 1;
        float mx = p[i][0];
#pragma unroll
        for (int j = 1; j < S; ++j) if (j <= jm) mx = fmaxf(mx, p[i][j]);
        float den = 0.f;
#pragma unroll
        for (int j = 0; j < S; ++j) if (j <= jm) { p[i][j] = __expf(p[i][j] - mx); den += p[i][j]; }
        const float inv = 1.f / den;
        float dot = 0.f;
#pragma unroll
        for (int j = 0; j < S; ++j) if (j <= jm) { p[i][j] *= inv; dot = fmaf(p[i][j], dp[i][j], dot); }
#pragma unroll
        for (int j = 0; j < S; ++j) if (j <= jm) dp[i][j] = p[i][j] * (dp[i][j] - dot) * scale;
    }
    // one output row at a time, so that only EPL accumulators are alive
#pragma unroll
    for (int s = 0; s < S; ++s) {
        T* base = dqkv + ((int64_t)b * S + s) * 3 * D + (int64_t)h * HD + l * EPL;
        float dq[EPL], dk[EPL], dv[EPL];
#pragma unroll
        for (int e = 0; e < EPL; ++e) { dq[e] = 0.f; dk[e] = 0.f; dv[e] = 0.f; }
#pragma unroll
        for (int t = 0; t < S; ++t) {
            if (!CAUSAL || t <= s) {
#pragma unroll
                for (int e = 0; e < EPL; ++e) dq[e] = fmaf(dp[s][t], k[t].get(e), dq[e]);
            }
            if (!CAUSAL || t >= s) {
#pragma unroll
                for (int e = 0; e < EPL; ++e) { dv[e] = fmaf(p[t][s], dO[t].get(e), dv[e]); dk[e] = fmaf(dp[t][s], q[t].get(e), dk[e]); }
            }
        }
        if (live) { LaneVec<T, EPL, VEC>::st(base, dq); LaneVec<T, EPL, VEC>::st(base + D, dk); LaneVec<T, EPL, VEC>::st(base + 2 * D, dv); }
    }
}

// ---------------------------------------------------------------------------------------------------- LayerNorm
// z = x (+ r); y = (z - mean) * rstd * gamma (+ beta).  One warp per row; rows of D <= 8192 elements.
// vec: all rows start on a multiple of four elements' size (widths are multiples of four), so four elements are one access.
// RMS = true is RMSNorm: the mean is taken as zero (y = z * rsqrt(mean(z^2) + eps) * gamma) and there is no beta.
template <typename T, bool RMS>
__global__ void __launch_bounds__(256) ln_fwd_kernel(const T* __restrict__ x, const T* __restrict__ r, const T* __restrict__ gamma,
                                                     const T* __restrict__ beta, T* __restrict__ z, T* __restrict__ y,
                                                     float* __restrict__ stats, int64_t rows, int D, float eps, bool vec) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const T* xr = x + row * D;
    const T* rr = r ? r + row * D : nullptr;
    float s = 0.f, ss = 0.f;
    for (int c = lane * 4; c < D; c += 128) {
        float a[4], bres[4];
        ld4<T>(xr, c, (D - c >= 4) ? 4 : D - c, vec, a);
        if (rr) { ld4<T>(rr, c, (D - c >= 4) ? 4 : D - c, vec, bres);
#pragma unroll
            for (int k = 0; k < 4; ++k) a[k] = Cvt<T>::to(Cvt<T>::from(a[k] + bres[k])); }
#pragma unroll
        for (int k = 0; k < 4; ++k) { s += a[k]; ss = fmaf(a[k], a[k], ss); }
    }
    s = warp_sum(s); ss = warp_sum(ss);
    const float mean = RMS ? 0.f : s / D;
    const float var = fmaxf(ss / D - mean * mean, 0.f);
    const float rstd = rsqrtf(var + eps);
    if (lane == 0) { stats[2 * row] = mean; stats[2 * row + 1] = rstd; }
    for (int c = lane * 4; c < D; c += 128) {
        const int cnt = (D - c >= 4) ? 4 : D - c;
        float a[4], bres[4], g[4], bb[4], o[4];
        ld4<T>(xr, c, cnt, vec, a);
        if (rr) { ld4<T>(rr, c, cnt, vec, bres);
#pragma unroll
            for (int k = 0; k < 4; ++k) a[k] = Cvt<T>::to(Cvt<T>::from(a[k] + bres[k]));
            st4<T>(z + row * D, c, cnt, vec, a); }
        ld4<T>(gamma, c, cnt, vec, g);
        if (beta) ld4<T>(beta, c, cnt, vec, bb);
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = (a[k] - mean) * rstd * g[k] + (beta ? bb[k] : 0.f);
        st4<T>(y + row * D, c, cnt, vec, o);
    }
}

// dz = rstd * (dy*g - mean_c(dy*g) - xhat * mean_c(dy*g*xhat)); per-CTA partial sums of dgamma / dbeta over its rows.
constexpr int LN_ROWS_PER_CTA = 64;
template <typename T, bool RMS>
__global__ void __launch_bounds__(256) ln_bwd_kernel(const T* __restrict__ z, const T* __restrict__ dy, const T* __restrict__ gamma,
                                                     const float* __restrict__ stats, const T* __restrict__ dz_in, T* __restrict__ dz,
                                                     float* __restrict__ part, int64_t rows, int D, bool vec) {
    extern __shared__ float sm[];                       // [8 warps][2][D]  per-warp column partials
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float* pg = sm + (size_t)w * 2 * D;
    float* pb = pg + D;
    for (int c = lane; c < D; c += 32) { pg[c] = 0.f; pb[c] = 0.f; }
    const int64_t row0 = (int64_t)blockIdx.x * LN_ROWS_PER_CTA;
    for (int rr = w; rr < LN_ROWS_PER_CTA; rr += 8) {
        const int64_t row = row0 + rr;
        if (row >= rows) break;
        const float mean = stats[2 * row], rstd = stats[2 * row + 1];
        float s1 = 0.f, s2 = 0.f;
        for (int c = lane * 4; c < D; c += 128) {
            const int cnt = (D - c >= 4) ? 4 : D - c;
            float a[4], d[4], g[4];
            ld4<T>(z + row * D, c, cnt, vec, a); ld4<T>(dy + row * D, c, cnt, vec, d); ld4<T>(gamma, c, cnt, vec, g);
#pragma unroll
            for (int k = 0; k < 4; ++k) if (k < cnt) {
                const float xh = (a[k] - mean) * rstd, dg = d[k] * g[k];
                s1 += dg; s2 = fmaf(dg, xh, s2);
                pg[c + k] = fmaf(d[k], xh, pg[c + k]); pb[c + k] += d[k];
            }
        }
        s1 = RMS ? 0.f : warp_sum(s1) / D; s2 = warp_sum(s2) / D;
        for (int c = lane * 4; c < D; c += 128) {
            const int cnt = (D - c >= 4) ? 4 : D - c;
            float a[4], d[4], g[4], o[4];
            ld4<T>(z + row * D, c, cnt, vec, a); ld4<T>(dy + row * D, c, cnt, vec, d); ld4<T>(gamma, c, cnt, vec, g);
#pragma unroll
            for (int k = 0; k < 4; ++k) { const float xh = (a[k] - mean) * rstd; o[k] = rstd * (d[k] * g[k] - s1 - xh * s2); }
            if (dz_in) {                                 // gradient that reached z directly (z is also the residual stream)
                float e[4];
                ld4<T>(dz_in + row * D, c, cnt, vec, e);
#pragma unroll
                for (int k = 0; k < 4; ++k) o[k] += e[k];
            }
            st4<T>(dz + row * D, c, cnt, vec, o);
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < D; c += 256) {
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int ww = 0; ww < 8; ++ww) { a += sm[(size_t)ww * 2 * D + c]; b += sm[(size_t)ww * 2 * D + D + c]; }
        part[((int64_t)blockIdx.x * 2) * D + c] = a;
        part[((int64_t)blockIdx.x * 2 + 1) * D + c] = b;
    }
}


// ---------------------------------------------------------------------------------------------------- whole 16-byte vectors
template <typename T> struct RowVec {
    static constexpr int VEC = 16 / sizeof(T);
    static __device__ __forceinline__ void get(const uint4 t, float (&v)[VEC]) {       // by value: through a reference to memory the elements are loaded one by one
        const T* h = reinterpret_cast<const T*>(&t);
#pragma unroll
        for (int k = 0; k < VEC; ++k) v[k] = Cvt<T>::to(h[k]);
    }
    static __device__ __forceinline__ uint4 put(const float (&v)[VEC]) {
        uint4 t;
        T* h = reinterpret_cast<T*>(&t);
#pragma unroll
        for (int k = 0; k < VEC; ++k) h[k] = Cvt<T>::from(v[k]);
        return t;
    }
};
template <typename T> __device__ __forceinline__ void row_ld(const T* p, float (&v)[RowVec<T>::VEC]) { RowVec<T>::get(*reinterpret_cast<const uint4*>(p), v); }
template <typename T> __device__ __forceinline__ void row_st(T* p, const float (&v)[RowVec<T>::VEC]) { *reinterpret_cast<uint4*>(p) = RowVec<T>::put(v); }

// Narrow rows of exactly NCH vectors per lane: a warp owns a row, so nothing has to be synchronised and no lane idles.
template <typename T, bool RMS, int NCH>
__global__ void __launch_bounds__(256) norm_fwd_wide_kernel(const T* __restrict__ x, const T* __restrict__ r, const T* __restrict__ gamma,
                                                            const T* __restrict__ beta, T* __restrict__ z, T* __restrict__ y,
                                                            float* __restrict__ stats, int64_t rows, float eps) {
    constexpr int VEC = RowVec<T>::VEC, D = 32 * VEC * NCH;
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    float a[NCH][VEC];
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
        const int col = (c * 32 + lane) * VEC;
        row_ld<T>(x + row * D + col, a[c]);
        if (r) {
            float b[VEC];
            row_ld<T>(r + row * D + col, b);
#pragma unroll
            for (int k = 0; k < VEC; ++k) a[c][k] = Cvt<T>::to(Cvt<T>::from(a[c][k] + b[k]));
            row_st<T>(z + row * D + col, a[c]);
        }
#pragma unroll
        for (int k = 0; k < VEC; ++k) { s += a[c][k]; ss = fmaf(a[c][k], a[c][k], ss); }
    }
    s = warp_sum(s); ss = warp_sum(ss);
    const float mean = RMS ? 0.f : s / D;
    const float rstd = rsqrtf(fmaxf(ss / D - mean * mean, 0.f) + eps);
    if (lane == 0) { stats[2 * row] = mean; stats[2 * row + 1] = rstd; }
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
        const int col = (c * 32 + lane) * VEC;
        float g[VEC], bb[VEC], o[VEC];
        row_ld<T>(gamma + col, g);
        if (beta) row_ld<T>(beta + col, bb);
#pragma unroll
        for (int k = 0; k < VEC; ++k) o[k] = (a[c][k] - mean) * rstd * g[k] + (beta ? bb[k] : 0.f);
        row_st<T>(y + row * D + col, o);
    }
}

template <typename T, bool RMS, int NCH>
__global__ void __launch_bounds__(256) norm_bwd_wide_kernel(const T* __restrict__ z, const T* __restrict__ dy, const T* __restrict__ gamma,
                                                            const float* __restrict__ stats, T* __restrict__ dz, float* __restrict__ part,
                                                            int64_t rows) {
    constexpr int VEC = RowVec<T>::VEC, D = 32 * VEC * NCH;
    extern __shared__ float sm[];                       // [8 warps][D]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float ag[NCH][VEC], ab[RMS ? 1 : NCH][VEC];        // gamma is re-read per row (4 KB, stays in L1): registers go to the accumulators
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int k = 0; k < VEC; ++k) { ag[c][k] = 0.f; if (!RMS) ab[c][k] = 0.f; }
    for (int64_t row = (int64_t)blockIdx.x * 8 + w; row < rows; row += (int64_t)gridDim.x * 8) {
        const float mean = stats[2 * row], rstd = stats[2 * row + 1];
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const int col = (c * 32 + lane) * VEC;
            float a[VEC], d[VEC], g[VEC];
            row_ld<T>(z + row * D + col, a); row_ld<T>(dy + row * D + col, d); row_ld<T>(gamma + col, g);
#pragma unroll
            for (int k = 0; k < VEC; ++k) { const float xh = (a[k] - mean) * rstd, dg = d[k] * g[k]; s1 += dg; s2 = fmaf(dg, xh, s2); }
        }
        s1 = RMS ? 0.f : warp_sum(s1) / D; s2 = warp_sum(s2) / D;
#pragma unroll
        for (int c = 0; c < NCH; ++c) {                 // second pass: the row is re-read through L1
            const int col = (c * 32 + lane) * VEC;
            float a[VEC], d[VEC], o[VEC], g[VEC];
            row_ld<T>(z + row * D + col, a); row_ld<T>(dy + row * D + col, d); row_ld<T>(gamma + col, g);
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
                const float xh = (a[k] - mean) * rstd;
                o[k] = rstd * (d[k] * g[k] - s1 - xh * s2);
                ag[c][k] = fmaf(d[k], xh, ag[c][k]);
                if (!RMS) ab[c][k] += d[k];
            }
            row_st<T>(dz + row * D + col, o);
        }
    }
    // fixed-order reduction over the eight warps, first the weight gradient, then (LayerNorm) the bias gradient
#pragma unroll 1
    for (int which = 0; which < (RMS ? 1 : 2); ++which) {
        __syncthreads();
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int k = 0; k < VEC; ++k) sm[w * D + (c * 32 + lane) * VEC + k] = which == 0 ? ag[c][k] : ab[RMS ? 0 : c][k];
        __syncthreads();
        for (int col = threadIdx.x; col < D; col += 256) {
            float acc = 0.f;
#pragma unroll
            for (int ww = 0; ww < 8; ++ww) acc += sm[ww * D + col];
            part[((int64_t)blockIdx.x * 2 + which) * D + col] = acc;
        }
    }
}

// Rows of any whole number of 16-byte vectors.  A row is spread over WPR = ceil(D / (32 VEC)) warps, one vector per lane, and a thread
// handles R rows at a time: all loads of the R rows (x and residual; z, dy and the residual stream's gradient) are in flight before the
// first is used, nothing is read or converted twice, and the backward keeps the weight (and bias) gradient of the thread's VEC columns in
// 2 VEC registers whatever the width.  A CTA holds G row groups of WPR warps; the row sums of a group's warps meet in shared memory.
// Bound by memory (268 MB each way at [16384, 2048] bf16 with residual: 41 us): RMSNorm forward 85 -> 45 us, backward 79 -> 49 us (one warp
// per row, eight vectors per lane); LayerNorm [8192, 3072] backward 371 -> 50 us, [32768, 768] 107 -> 44 us (the four-wide general kernels,
// which took every width that is not a power of two).
constexpr int NORM_MAX_WPR = 24, NORM_R4_WPR = 8;      // 3072 fp32 columns; four rows per thread need the registers of a smaller CTA

// sums a[0..N) over the wpr warps of this thread's row group; `buf` is [warps][N].  The warps' sums are added in a tree: one after the
// other, the last of 24 additions of squares would round at the size of the whole sum.
template <int N>
__device__ __forceinline__ void group_totals(float (&a)[N], int wpr, float* buf) {
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = warp_sum(a[i]);
    if (wpr == 1) return;
    const int w = threadIdx.x >> 5, w0 = w - w % wpr;
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int i = 0; i < N; ++i) buf[w * N + i] = a[i];
    __syncthreads();
    const int span = 2 << (31 - __clz(wpr - 1)), k = threadIdx.x & (span - 1);       // power of two that holds wpr >= 2 warps
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = k < wpr ? buf[(w0 + k) * N + i] : 0.f;
    for (int o = span >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) a[i] += __shfl_xor_sync(0xffffffffu, a[i], o);
}

template <typename T, bool RMS, int R>
__global__ void __launch_bounds__(R == 1 ? 32 * NORM_MAX_WPR : 32 * NORM_R4_WPR, R == 1 ? 1 : 3) norm_fwd_vec_kernel(const T* __restrict__ x, const T* __restrict__ r, const T* __restrict__ gamma,
                                                                        const T* __restrict__ beta, T* __restrict__ z, T* __restrict__ y,
                                                                        float* __restrict__ stats, int64_t rows, int D, int wpr, float eps) {
    constexpr int VEC = RowVec<T>::VEC;
    __shared__ float sums[NORM_MAX_WPR][2 * R];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = w % wpr, groups = (blockDim.x >> 5) / wpr;
    const int col = (c * 32 + lane) * VEC;
    const int64_t row0 = ((int64_t)blockIdx.x * groups + w / wpr) * R;
    const bool in = col < D;
    uint4 xv[R], rv[R];
    bool ok[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        ok[i] = in && row0 + i < rows;
        xv[i] = rv[i] = make_uint4(0, 0, 0, 0);
        if (ok[i]) {
            xv[i] = *reinterpret_cast<const uint4*>(x + (row0 + i) * D + col);
            if (r) rv[i] = *reinterpret_cast<const uint4*>(r + (row0 + i) * D + col);
        }
    }
    float t[2 * R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        float a[VEC];
        RowVec<T>::get(xv[i], a);
        if (r) {
            float b[VEC];
            RowVec<T>::get(rv[i], b);
#pragma unroll
            for (int k = 0; k < VEC; ++k) a[k] += b[k];
            xv[i] = RowVec<T>::put(a);
            if (ok[i]) *reinterpret_cast<uint4*>(z + (row0 + i) * D + col) = xv[i];
            RowVec<T>::get(xv[i], a);                     // the sum as it is stored
        }
        float s = 0.f, ss = 0.f;
#pragma unroll
        for (int k = 0; k < VEC; ++k) { s += a[k]; ss = fmaf(a[k], a[k], ss); }
        t[2 * i] = s; t[2 * i + 1] = ss;
    }
    group_totals<2 * R>(t, wpr, &sums[0][0]);
    float g[VEC], bb[VEC];
    if (in) {
        RowVec<T>::get(*reinterpret_cast<const uint4*>(gamma + col), g);
        if (beta) RowVec<T>::get(*reinterpret_cast<const uint4*>(beta + col), bb);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (!ok[i]) continue;
        const float mean = RMS ? 0.f : t[2 * i] / D;
        const float rstd = rsqrtf(fmaxf(t[2 * i + 1] / D - mean * mean, 0.f) + eps);
        if (c == 0 && lane == 0) *reinterpret_cast<float2*>(stats + 2 * (row0 + i)) = make_float2(mean, rstd);
        float a[VEC], o[VEC];
        RowVec<T>::get(xv[i], a);
#pragma unroll
        for (int k = 0; k < VEC; ++k) o[k] = RMS ? a[k] * rstd * g[k] : fmaf((a[k] - mean) * rstd, g[k], beta ? bb[k] : 0.f);
        *reinterpret_cast<uint4*>(y + (row0 + i) * D + col) = RowVec<T>::put(o);
    }
}

template <typename T, bool RMS, int R>
__global__ void __launch_bounds__(R == 1 ? 32 * NORM_MAX_WPR : 32 * NORM_R4_WPR, R == 1 ? 1 : 2) norm_bwd_vec_kernel(const T* __restrict__ z, const T* __restrict__ dy, const T* __restrict__ gamma,
                                                                        const float* __restrict__ stats, const T* __restrict__ dz_in, T* __restrict__ dz,
                                                                        float* __restrict__ part, int64_t rows, int D, int wpr) {
    constexpr int VEC = RowVec<T>::VEC;
    __shared__ float sums[2][NORM_MAX_WPR][2 * R];
    __shared__ float red[8][32 * VEC];                    // used when several row groups share a CTA (at most 8 warps then)
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = w % wpr, groups = (blockDim.x >> 5) / wpr;
    const int col = (c * 32 + lane) * VEC;
    const bool in = col < D;
    // Parameter gradients of this thread's columns: the R rows of a round are summed first (R > 1), or the sums of eight rounds (R = 1), so
    // that a long call does not add its rows one by one to a sum that outgrows them.
    float g[VEC], ag[VEC], ab[VEC], bg[VEC], bb[VEC];
#pragma unroll
    for (int k = 0; k < VEC; ++k) g[k] = ag[k] = ab[k] = bg[k] = bb[k] = 0.f;
    if (in) RowVec<T>::get(*reinterpret_cast<const uint4*>(gamma + col), g);
    int rounds = 0;
    const int64_t step = (int64_t)gridDim.x * groups * R;
    const float inv_d = 1.f / D;
    int par = 0;
    for (int64_t base = (int64_t)blockIdx.x * groups * R; base < rows; base += step, par ^= 1) {
        const int64_t row0 = base + (w / wpr) * R;
        uint4 zv[R], dv[R], ev[R];
        float2 st[R];
        bool ok[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            ok[i] = in && row0 + i < rows;
            zv[i] = dv[i] = ev[i] = make_uint4(0, 0, 0, 0);
            st[i] = make_float2(0.f, 0.f);
            if (ok[i]) {
                st[i] = *reinterpret_cast<const float2*>(stats + 2 * (row0 + i));
                zv[i] = *reinterpret_cast<const uint4*>(z + (row0 + i) * D + col);
                dv[i] = *reinterpret_cast<const uint4*>(dy + (row0 + i) * D + col);
                if (dz_in) ev[i] = *reinterpret_cast<const uint4*>(dz_in + (row0 + i) * D + col);
            }
        }
        float t[2 * R], xh[R][VEC], dg[R][VEC];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float d[VEC];
            RowVec<T>::get(zv[i], xh[i]); RowVec<T>::get(dv[i], d);
            float s1 = 0.f, s2 = 0.f;
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
                xh[i][k] = (RMS ? xh[i][k] : xh[i][k] - st[i].x) * st[i].y;
                dg[i][k] = d[k] * g[k];
                if (!RMS) s1 += dg[i][k];
                s2 = fmaf(dg[i][k], xh[i][k], s2);
                bg[k] = fmaf(d[k], xh[i][k], bg[k]);
                if (!RMS) bb[k] += d[k];
            }
            if constexpr (RMS) t[i] = s2;
            else { t[2 * i] = s1; t[2 * i + 1] = s2; }
        }
        if (R > 1 || (++rounds & 7) == 0) {
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
                ag[k] += bg[k]; bg[k] = 0.f;
                if (!RMS) { ab[k] += bb[k]; bb[k] = 0.f; }
            }
        }
        if constexpr (RMS) {
            float u[R];
#pragma unroll
            for (int i = 0; i < R; ++i) u[i] = t[i];
            group_totals<R>(u, wpr, &sums[par][0][0]);    // two buffers: the next round's sums may be written while these are read
#pragma unroll
            for (int i = R - 1; i >= 0; --i) { t[2 * i + 1] = u[i]; t[2 * i] = 0.f; }
        } else group_totals<2 * R>(t, wpr, &sums[par][0][0]);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (!ok[i]) continue;
            const float rs = st[i].y, c1 = RMS ? 0.f : -rs * (t[2 * i] * inv_d), c2 = -rs * (t[2 * i + 1] * inv_d);
            float o[VEC];
#pragma unroll
            for (int k = 0; k < VEC; ++k) o[k] = fmaf(dg[i][k], rs, RMS ? xh[i][k] * c2 : fmaf(xh[i][k], c2, c1));
            if (dz_in) {                                  // gradient that reached z directly (z is also the residual stream)
                float e[VEC];
                RowVec<T>::get(ev[i], e);
#pragma unroll
                for (int k = 0; k < VEC; ++k) o[k] += e[k];
            }
            *reinterpret_cast<uint4*>(dz + (row0 + i) * D + col) = RowVec<T>::put(o);
        }
    }
    // the CTA's partial sums of the weight and (LayerNorm) bias gradient: row groups added in order
    for (int which = 0; which < (RMS ? 1 : 2); ++which) {
        float v[VEC];
#pragma unroll
        for (int k = 0; k < VEC; ++k) v[k] = which == 0 ? ag[k] + bg[k] : ab[k] + bb[k];
        if (groups > 1) {
            __syncthreads();
#pragma unroll
            for (int k = 0; k < VEC; ++k) red[w][lane * VEC + k] = v[k];
            __syncthreads();
            if (w >= wpr) continue;
            for (int q = 1; q < groups; ++q)
#pragma unroll
                for (int k = 0; k < VEC; ++k) v[k] += red[w + q * wpr][lane * VEC + k];
        }
        if (in) {
            float* o = part + ((int64_t)blockIdx.x * 2 + which) * D + col;
#pragma unroll
            for (int k = 0; k < VEC; k += 4) *reinterpret_cast<float4*>(o + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
        }
    }
}

// Second stage of the parameter gradients: column c of dgamma / dbeta is the sum of its n_part partial rows.  A CTA owns 32
// columns; its 32 warps take the partial rows p = warp, warp + 32, ... and the 32 sub-sums are added in a tree, so the
// result does not depend on timing.  (D / 32 CTAs only: with 8 warps per CTA the kernel took 9 us for 296 partial rows of 512 columns.)
constexpr int LN_RED_WARPS = 32;
template <typename T>
__global__ void __launch_bounds__(32 * LN_RED_WARPS) ln_bwd_reduce_kernel(const float* __restrict__ part, int n_part, int D, T* __restrict__ dgamma,
                                                                          T* __restrict__ dbeta, bool accumulate) {
    __shared__ float sh[2][LN_RED_WARPS][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    float a = 0.f, b = 0.f;
    if (c < D) {
        int p = w;
        for (; p + 3 * LN_RED_WARPS < n_part; p += 4 * LN_RED_WARPS) {
            float va[4], vb[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                va[u] = part[((int64_t)(p + LN_RED_WARPS * u) * 2) * D + c];
                vb[u] = dbeta ? part[((int64_t)(p + LN_RED_WARPS * u) * 2 + 1) * D + c] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) { a += va[u]; b += vb[u]; }
        }
        for (; p < n_part; p += LN_RED_WARPS) { a += part[((int64_t)p * 2) * D + c]; if (dbeta) b += part[((int64_t)p * 2 + 1) * D + c]; }
    }
    sh[0][w][lane] = a; sh[1][w][lane] = b;
    __syncthreads();
    // warp w adds the 32 sub-sums of column w in a tree
    a = warp_sum(sh[0][lane][w]); b = warp_sum(sh[1][lane][w]);
    const int col = blockIdx.x * 32 + w;
    if (lane == 0 && col < D) {
        // accumulate: dgamma / dbeta are the parameters' gradient buffers and already hold other contributions of this step
        if (accumulate) { a += Cvt<T>::to(dgamma[col]); if (dbeta) b += Cvt<T>::to(dbeta[col]); }
        dgamma[col] = Cvt<T>::from(a);
        if (dbeta) dbeta[col] = Cvt<T>::from(b);
    }
}

}  // namespace

bool attn_small_supported(int S, int HD) { return (S == 4 || S == 8) && (HD == 32 || HD == 64); }

static bool aligned(const void* p, size_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }
static bool aligned16(const void* p) { return aligned(p, 16); }

template <typename T>
static void attn_dispatch(bool bwd, const T* qkv, const T* dout, T* out, int B, int S, int H, int HD, bool causal, cudaStream_t st) {
    const float scale = 1.f / sqrtf((float)HD);
    if ((int64_t)B * H == 0) return;
    count_launch();
#define GO(SV, EV, HV, CV, VV) { \
    const unsigned blocks = (unsigned)(((int64_t)B * H + 128 / (HV / EV) - 1) / (128 / (HV / EV))); \
    if (bwd) attn_small_bwd_kernel<T, SV, EV, HV, CV, VV><<<blocks, 128, 0, st>>>(qkv, dout, out, B, H, scale); \
    else attn_small_fwd_kernel<T, SV, EV, HV, CV, VV><<<blocks, 128, 0, st>>>(qkv, out, B, H, scale); }
#define GO2(SV, EV, HV, VV) { if (causal) GO(SV, EV, HV, true, VV) else GO(SV, EV, HV, false, VV) }
    // Sixteen bytes per lane; half of that for eight positions, whose scores and rows need the registers.  A storage offset that breaks
    // the alignment (a view into a larger buffer, at any element) takes a warp per head and loads element by element.
    constexpr int V4 = 16 / (int)sizeof(T), V8 = 8 / (int)sizeof(T);
    const bool al = aligned16(qkv) && aligned16(dout) && aligned16(out);
    if (al && S == 4) { if (HD == 64) GO2(4, V4, 64, true) else GO2(4, V4, 32, true) }
    else if (al) { if (HD == 64) GO2(8, V8, 64, true) else GO2(8, V8, 32, true) }
    else if (S == 4) { if (HD == 64) GO2(4, 2, 64, false) else GO2(4, 1, 32, false) }
    else { if (HD == 64) GO2(8, 2, 64, false) else GO2(8, 1, 32, false) }
#undef GO2
#undef GO
}

void attn_small(int dtype, bool bwd, const void* qkv, const void* dout, void* out, int B, int S, int H, int HD, bool causal, cudaStream_t st) {
    if (dtype == BF16) attn_dispatch<__nv_bfloat16>(bwd, (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)dout, (__nv_bfloat16*)out, B, S, H, HD, causal, st);
    else attn_dispatch<float>(bwd, (const float*)qkv, (const float*)dout, (float*)out, B, S, H, HD, causal, st);
}

// The vector kernels take rows of whole 16-byte vectors: WPR warps per row, 8 / WPR row groups per CTA.  0: the row does not qualify.
static int norm_wpr(int D, int elem_bytes) {
    const int vec = 16 / elem_bytes;
    if (D % vec) return 0;
    const int wpr = (D + 32 * vec - 1) / (32 * vec);
    return wpr <= NORM_MAX_WPR ? wpr : 0;
}
// Rows of exactly 32 lanes x {1, 2, 4} vectors may take a warp each (no synchronisation between warps).  Measured, us, warp per row against
// warps per row: forward with residual [32768, 512] bf16 20.9 : 26.9, [8192, 512] fp32 11.1 : 12.9, [32768, 1024] bf16 57.8 : 50.3; backward
// without a third input [32768, 512] 23.5 : 27.0, [32768, 1024] 47.8 : 53.2, fp32 8.2 : 11.9, with one [32768, 256] 20.7 : 13.3 and
// [32768, 1024] 103 : 48.7.
static bool norm_warp_rows(int D, int wpr, int elem_bytes, int max_wpr) { return wpr <= max_wpr && wpr != 3 && D == 32 * (16 / elem_bytes) * wpr; }

struct NormShape { int threads, rows_per_cta, r; };
// Four rows per thread keep enough loads in flight; a call with few rows spreads them over more CTAs, one row per thread.
static NormShape norm_shape(int64_t rows, int wpr) {
    const int groups = wpr < 8 ? 8 / wpr : 1;
    const int r = wpr <= NORM_R4_WPR && rows >= (int64_t)148 * 2 * groups * 4 ? 4 : 1;
    return {32 * wpr * groups, groups * r, r};
}

template <typename T>
static void ln_fwd_t(bool rms, const void* x, const void* r, const void* gamma, const void* beta, void* z, void* y, float* stats, int64_t rows, int D,
                     float eps, cudaStream_t st) {
    const int wpr = norm_wpr(D, (int)sizeof(T));
    if (wpr && aligned16(x) && aligned16(r) && aligned16(gamma) && aligned16(beta) && aligned16(z) && aligned16(y)) {
        if (norm_warp_rows(D, wpr, (int)sizeof(T), sizeof(T) == 2 ? 2 : 4)) {
            const unsigned g8 = (unsigned)((rows + 7) / 8);
#define WIDE_F(N) \
            if (rms) norm_fwd_wide_kernel<T, true, N><<<g8, 256, 0, st>>>((const T*)x, (const T*)r, (const T*)gamma, nullptr, (T*)z, (T*)y, stats, rows, eps); \
            else norm_fwd_wide_kernel<T, false, N><<<g8, 256, 0, st>>>((const T*)x, (const T*)r, (const T*)gamma, (const T*)beta, (T*)z, (T*)y, stats, rows, eps);
            switch (wpr) { case 1: WIDE_F(1) break; case 2: WIDE_F(2) break; default: if constexpr (sizeof(T) == 4) { WIDE_F(4) } }      // 16 bits stop at two
#undef WIDE_F
            return;
        }
        const NormShape sh = norm_shape(rows, wpr);
        const unsigned grid = (unsigned)((rows + sh.rows_per_cta - 1) / sh.rows_per_cta);
#define VEC_F(RMS, RR) norm_fwd_vec_kernel<T, RMS, RR><<<grid, sh.threads, 0, st>>>((const T*)x, (const T*)r, (const T*)gamma, RMS ? nullptr : (const T*)beta, \
                                                                                   (T*)z, (T*)y, stats, rows, D, wpr, eps)
        if (rms) { if (sh.r > 1) VEC_F(true, 4); else VEC_F(true, 1); }
        else { if (sh.r > 1) VEC_F(false, 4); else VEC_F(false, 1); }
#undef VEC_F
        return;
    }
    const unsigned blocks = (unsigned)((rows + 7) / 8);
    constexpr size_t A = 4 * sizeof(T);
    const bool vec = aligned(x, A) && aligned(r, A) && aligned(gamma, A) && aligned(beta, A) && aligned(z, A) && aligned(y, A);
    if (rms) ln_fwd_kernel<T, true><<<blocks, 256, 0, st>>>((const T*)x, (const T*)r, (const T*)gamma, nullptr, (T*)z, (T*)y, stats, rows, D, eps, vec);
    else ln_fwd_kernel<T, false><<<blocks, 256, 0, st>>>((const T*)x, (const T*)r, (const T*)gamma, (const T*)beta, (T*)z, (T*)y, stats, rows, D, eps, vec);
}

void ln_fwd(int dtype, bool rms, const void* x, const void* r, const void* gamma, const void* beta, void* z, void* y, float* stats, int64_t rows,
            int D, float eps, cudaStream_t st) {
    count_launch();
    if (dtype == BF16) ln_fwd_t<__nv_bfloat16>(rms, x, r, gamma, beta, z, y, stats, rows, D, eps, st);
    else ln_fwd_t<float>(rms, x, r, gamma, beta, z, y, stats, rows, D, eps, st);
}

// CTA partials of the weight / bias gradient: enough for either backward kernel
constexpr int NORM_BWD_GRID = 148 * 2;
int ln_bwd_parts(int64_t rows) {
    const int a = (int)((rows + LN_ROWS_PER_CTA - 1) / LN_ROWS_PER_CTA), b = (int)(rows < NORM_BWD_GRID ? rows : NORM_BWD_GRID);
    return a > b ? a : b > 1 ? b : 1;
}

template <typename T>
static void ln_bwd_t(bool rms, const void* z, const void* dy, const void* gamma, const float* stats, const void* dz_in, void* dz, float* part,
                     void* dgamma, void* dbeta, bool accumulate, int64_t rows, int D, cudaStream_t st) {
    const int wpr = norm_wpr(D, (int)sizeof(T));
    if (wpr && aligned16(z) && aligned16(dy) && aligned16(gamma) && aligned16(dz_in) && aligned16(dz)) {
        if (dz_in == nullptr && norm_warp_rows(D, wpr, (int)sizeof(T), 4)) {
            const int64_t n8 = (rows + 7) / 8;
            const int g8 = (int)(n8 < 1 ? 1 : n8 < NORM_BWD_GRID ? n8 : NORM_BWD_GRID);
            const size_t smw = (size_t)8 * D * sizeof(float);
#define WIDE_B(N) \
            if (rms) norm_bwd_wide_kernel<T, true, N><<<g8, 256, smw, st>>>((const T*)z, (const T*)dy, (const T*)gamma, stats, (T*)dz, part, rows); \
            else norm_bwd_wide_kernel<T, false, N><<<g8, 256, smw, st>>>((const T*)z, (const T*)dy, (const T*)gamma, stats, (T*)dz, part, rows);
            switch (wpr) { case 1: WIDE_B(1) break; case 2: WIDE_B(2) break; default: WIDE_B(4) }
#undef WIDE_B
            ln_bwd_reduce_kernel<T><<<(D + 31) / 32, 32 * LN_RED_WARPS, 0, st>>>(part, g8, D, (T*)dgamma, (T*)dbeta, accumulate);
            return;
        }
        const NormShape sh = norm_shape(rows, wpr);
        const int64_t need = (rows + sh.rows_per_cta - 1) / sh.rows_per_cta;
        const int grid = (int)(need < 1 ? 1 : need < NORM_BWD_GRID ? need : NORM_BWD_GRID);
#define VEC_B(RMS, RR) norm_bwd_vec_kernel<T, RMS, RR><<<grid, sh.threads, 0, st>>>((const T*)z, (const T*)dy, (const T*)gamma, stats, (const T*)dz_in, (T*)dz, part, rows, D, wpr)
        if (rms) { if (sh.r > 1) VEC_B(true, 4); else VEC_B(true, 1); }
        else { if (sh.r > 1) VEC_B(false, 4); else VEC_B(false, 1); }
#undef VEC_B
        ln_bwd_reduce_kernel<T><<<(D + 31) / 32, 32 * LN_RED_WARPS, 0, st>>>(part, grid, D, (T*)dgamma, (T*)dbeta, accumulate);
        return;
    }
    const int parts = (int)((rows + LN_ROWS_PER_CTA - 1) / LN_ROWS_PER_CTA);
    const size_t smem = (size_t)8 * 2 * D * sizeof(float);
    constexpr size_t A = 4 * sizeof(T);
    const bool vec = aligned(z, A) && aligned(dy, A) && aligned(gamma, A) && aligned(dz_in, A) && aligned(dz, A);
    if (rms) {
        cudaFuncSetAttribute(ln_bwd_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        ln_bwd_kernel<T, true><<<parts, 256, smem, st>>>((const T*)z, (const T*)dy, (const T*)gamma, stats, (const T*)dz_in, (T*)dz, part, rows, D, vec);
    } else {
        cudaFuncSetAttribute(ln_bwd_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        ln_bwd_kernel<T, false><<<parts, 256, smem, st>>>((const T*)z, (const T*)dy, (const T*)gamma, stats, (const T*)dz_in, (T*)dz, part, rows, D, vec);
    }
    ln_bwd_reduce_kernel<T><<<(D + 31) / 32, 32 * LN_RED_WARPS, 0, st>>>(part, parts, D, (T*)dgamma, (T*)dbeta, accumulate);
}

void ln_bwd(int dtype, bool rms, const void* z, const void* dy, const void* gamma, const float* stats, const void* dz_in, void* dz, float* part,
            void* dgamma, void* dbeta, bool accumulate, int64_t rows, int D, cudaStream_t st) {
    count_launch(2);
    if (dtype == BF16) ln_bwd_t<__nv_bfloat16>(rms, z, dy, gamma, stats, dz_in, dz, part, dgamma, dbeta, accumulate, rows, D, st);
    else ln_bwd_t<float>(rms, z, dy, gamma, stats, dz_in, dz, part, dgamma, dbeta, accumulate, rows, D, st);
}


// ---------------------------------------------------------------------------------------------------------------------------
// Column sums of a row-major [rows, C] matrix: the bias gradient of a Linear layer (db = sum over tokens of dy).  Two stages in
// a fixed order (no atomics): CTA (bx, by) sums rows [by * rows_per_cta, ...) of a slab of 32 sixteen-byte vectors, eight row
// lanes per column vector with fp32 accumulators, and writes one partial row; the second kernel adds the partial rows in order.
namespace {
template <typename T>
__global__ void __launch_bounds__(256) col_sum_part_kernel(const T* __restrict__ x, int64_t ld, int64_t rows, int C, int64_t rows_per_cta,
                                                           bool vec, float* __restrict__ part) {
    constexpr int VEC = 16 / (int)sizeof(T);
    __shared__ float sh[8][32 * VEC + 1];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int c0 = (blockIdx.x * 32 + tx) * VEC;
    const int64_t r0 = (int64_t)blockIdx.y * rows_per_cta;
    const int64_t r1 = r0 + rows_per_cta < rows ? r0 + rows_per_cta : rows;
    // sub: the sum of up to 32 rows, added to acc at a time, so that a long chain of rows does not round at the size of its sum
    float acc[VEC], sub[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) acc[j] = sub[j] = 0.f;
    const auto flush = [&] {
#pragma unroll
        for (int j = 0; j < VEC; ++j) { acc[j] += sub[j]; sub[j] = 0.f; }
    };
    if (c0 < C) {
        if (vec) {
            int64_t r = r0 + ty;
            for (int n = 1; r + 24 < r1; r += 32, ++n) {      // four independent 16-byte loads in flight per thread
                uint4 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const uint4*>(x + (r + 8 * u) * ld + c0);
                const T *e0 = reinterpret_cast<const T*>(&v[0]), *e1 = reinterpret_cast<const T*>(&v[1]), *e2 = reinterpret_cast<const T*>(&v[2]),
                        *e3 = reinterpret_cast<const T*>(&v[3]);
#pragma unroll
                for (int j = 0; j < VEC; ++j) sub[j] += (Cvt<T>::to(e0[j]) + Cvt<T>::to(e1[j])) + (Cvt<T>::to(e2[j]) + Cvt<T>::to(e3[j]));
                if ((n & 7) == 0) flush();
            }
            for (; r < r1; r += 8) {
                const uint4 v = *reinterpret_cast<const uint4*>(x + r * ld + c0);
                const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
                for (int j = 0; j < VEC; ++j) sub[j] += Cvt<T>::to(e[j]);
            }
        } else {
            for (int64_t r = r0 + ty, n = 1; r < r1; r += 8, ++n) {
#pragma unroll
                for (int j = 0; j < VEC; ++j)
                    if (c0 + j < C) sub[j] += Cvt<T>::to(x[r * ld + c0 + j]);
                if ((n & 15) == 0) flush();
            }
        }
        flush();
    }
#pragma unroll
    for (int j = 0; j < VEC; ++j) sh[ty][tx * VEC + j] = acc[j];
    __syncthreads();
    for (int c = threadIdx.x; c < 32 * VEC; c += 256) {
        const int col = blockIdx.x * 32 * VEC + c;
        if (col < C) {
            part[(int64_t)blockIdx.y * C + col] = ((sh[0][c] + sh[1][c]) + (sh[2][c] + sh[3][c])) + ((sh[4][c] + sh[5][c]) + (sh[6][c] + sh[7][c]));
        }
    }
}

// Second stage: 32 columns per CTA; warp w adds the partial rows w, w + 8, ... and the 8 sub-sums are added in a tree.
template <typename T>
__global__ void __launch_bounds__(256) col_sum_final_kernel(const float* __restrict__ part, int parts, int C, T* __restrict__ out,
                                                            bool accumulate) {
    __shared__ float sh[8][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    float t = 0.f;
    if (c < C) {
        int p = w;
        for (; p + 24 < parts; p += 32) {
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = part[(int64_t)(p + 8 * u) * C + c];
            t += (v[0] + v[1]) + (v[2] + v[3]);
        }
        for (; p < parts; p += 8) t += part[(int64_t)p * C + c];
    }
    sh[w][lane] = t;
    __syncthreads();
    if (w == 0 && c < C) {
        t = ((sh[0][lane] + sh[1][lane]) + (sh[2][lane] + sh[3][lane])) + ((sh[4][lane] + sh[5][lane]) + (sh[6][lane] + sh[7][lane]));
        if (accumulate) t += Cvt<T>::to(out[c]);
        out[c] = Cvt<T>::from(t);
    }
}
}  // namespace

// number of partial rows the first stage writes for a [rows, C] input (the caller provides parts * C floats of scratch)
int col_sum_parts(int64_t rows, int C, int elem_bytes) {
    const int vecw = 32 * (16 / elem_bytes);
    const int bx = (C + vecw - 1) / vecw;
    int64_t parts = (4 * 148 + bx - 1) / bx;
    const int64_t max_parts = (rows + 63) / 64;
    if (parts > max_parts) parts = max_parts;
    return parts < 1 ? 1 : (int)parts;
}

void col_sum(int dtype, const void* x, int64_t ld, int64_t rows, int C, float* part, void* out, bool accumulate, cudaStream_t st) {
    const int es = dtype == F32 ? 4 : 2;
    const int parts = col_sum_parts(rows, C, es);
    const int64_t rpc = (rows + parts - 1) / parts;
    const int vecw = 32 * (16 / es);
    const dim3 grid((C + vecw - 1) / vecw, parts);
    const bool vec = C % (16 / es) == 0 && (ld * es) % 16 == 0 && aligned16(x);
    count_launch(2);
    if (dtype == BF16) {
        col_sum_part_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)x, ld, rows, C, rpc, vec, part);
        col_sum_final_kernel<__nv_bfloat16><<<(C + 31) / 32, 256, 0, st>>>(part, parts, C, (__nv_bfloat16*)out, accumulate);
    } else if (dtype == F16) {
        col_sum_part_kernel<__half><<<grid, 256, 0, st>>>((const __half*)x, ld, rows, C, rpc, vec, part);
        col_sum_final_kernel<__half><<<(C + 31) / 32, 256, 0, st>>>(part, parts, C, (__half*)out, accumulate);
    } else {
        col_sum_part_kernel<float><<<grid, 256, 0, st>>>((const float*)x, ld, rows, C, rpc, vec, part);
        col_sum_final_kernel<float><<<(C + 31) / 32, 256, 0, st>>>(part, parts, C, (float*)out, accumulate);
    }
}

}  // namespace sg
