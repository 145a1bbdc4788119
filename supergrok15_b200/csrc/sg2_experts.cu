// Routed expert evaluation of the SuperGrok v2 bilevel (soft top-k) path, forward and backward (sm_100a).
//
// After the product-key routing every head of an element holds 4 row keys (ia, weight wa) and 4 column keys (ib, wb); the 16
// experts e = ia*pk + ib are evaluated on the element's scalar gradient g with weight wa*wb:
//     total[n] = sum_h sum_a sum_b wa[n,h,a] * wb[n,h,b] * expert_e(g[n]),   expert_e(g) = b2[e] + sum_j relu(g*W1[e,j] + b1[e,j]) * W2[e,j]
// The PyTorch formulation of this step (reference grokking_optimizers/supergrok2.py:717-807 evaluates it per head with
// gathered expert weights; a dense variant evaluates all 144 experts for every element) materialises [n, 144, 16] tensors in
// the forward and the backward pass; here nothing but the routing tables crosses HBM.
//
// Backward: d wa / d wb per element, and the expert-parameter gradients summed over all elements WITHOUT atomics: a tile of
// elements first scatters dtotal*wa*wb into a dense [elements, experts] table in shared memory (head after head, so the
// order of additions is fixed), then every thread owns up to nine fixed (expert, hidden unit) pairs - their weights in
// registers - and walks the tile's elements; per-CTA sums go to a partial buffer that a second kernel adds in CTA order.
#include "sg_native.h"
#include "column_parts.cuh"

namespace sg {
namespace {

constexpr int XH = 16;            // expert hidden width
constexpr int XK = 4;             // keys kept per sub-key (top-4 x top-4 = 16 experts per head)
constexpr int XTHREADS = 256;
constexpr int XMAXQ = 9;          // (expert, hidden) pairs per thread in the backward pass: experts <= 16 * XMAXQ = 144
constexpr int XE = 16 * XMAXQ;    // row pitch of the dense routing table (columns from E on stay zero)
constexpr int XSEG = XH + 1;      // linear pieces of an expert = row pitch of its tables (odd: different experts fall into different banks)

// An expert is a piecewise linear function of the scalar g: hidden unit j switches at t_j = -b1_j / W1_j.  The tables hold the sorted
// switching points and, per piece, slope and intercept (summed in fp64), so that a value takes five comparisons and a compensated
// multiply-add instead of 16 hidden units with three table words each; both forms are bound by the shared-memory reads (54 against 9 words
// per value).  Forward at 422,755 elements 385 us with units, 113 us with the table.
// slope * g and the intercept cancel where g lies near the switching points of the units that are on: each unit then has a small value,
// which the sum over the units rounds relative to itself.  So slope and intercept are pairs of floats (value and remainder) and the
// product and the sum keep their rounding errors: what is lost is 2^-47 of |slope * g|.  (Plain floats take 81 us and are 8e-6 off with
// all switching points within 1e-4 of the gradients, where the units are 6e-8 off.)  The switching points are rounded towards
// -infinity: for every float g, g > t_j then decides exactly as the sign of g * W1_j + b1_j does.
struct XTable { const float4* v; const float* t; };                            // v: slope, its remainder, intercept, its remainder
size_t __host__ __device__ constexpr x_table_floats(int E) { return (size_t)E * XSEG * 5; }

// sixteen lanes per expert: lane j ranks its switching point, lane s sums piece s (lane 0 also piece 16)
__global__ void __launch_bounds__(128) experts_table_kernel(const float* __restrict__ W1, const float* __restrict__ b1, const float* __restrict__ W2,
                                                            const float* __restrict__ b2, int E, float* __restrict__ table) {
    const int e_raw = blockIdx.x * 8 + (threadIdx.x >> 4), j = threadIdx.x & 15;
    const int e = e_raw < E ? e_raw : E - 1;                          // whole warps take part in the shuffles
    float w1 = W1[e * XH + j], b = b1[e * XH + j];
    const float w2 = W2[e * XH + j];
    if (isnan(w1) || isnan(b)) w1 = b = 0.f;                           // such a unit is off, as fmaxf(NaN, 0) makes it; the ranks below have to be distinct
    const float t = w1 != 0.f ? __fdiv_rd(-b, w1) : INFINITY;
    int rank = 0;
    for (int k = 0; k < XH; ++k) {
        const float tk = __shfl_sync(0xffffffffu, t, k, 16);
        rank += (tk < t || (tk == t && k < j)) ? 1 : 0;
    }
    float4* val = reinterpret_cast<float4*>(table) + (size_t)e * XSEG;
    float* th = table + 4 * (size_t)E * XSEG + (size_t)e * XSEG;
    if (e_raw < E) th[rank] = t;
    const double base = (double)b2[e];
    for (int rep = 0; rep < 2; ++rep) {
        const int s = rep == 0 ? j : XH;                               // piece s: the s lowest switching points lie below g
        double slope = 0.0, icept = base;
        for (int k = 0; k < XH; ++k) {
            const float kw1 = __shfl_sync(0xffffffffu, w1, k, 16), kb = __shfl_sync(0xffffffffu, b, k, 16), kw2 = __shfl_sync(0xffffffffu, w2, k, 16);
            const int kr = __shfl_sync(0xffffffffu, rank, k, 16);
            const bool on = kw1 > 0.f ? kr < s : kw1 < 0.f ? kr >= s : kb > 0.f;
            if (on) { slope += (double)kw2 * kw1; icept += (double)kw2 * kb; }
            else icept += 0.0 * kw2;                                   // a non-finite W2 shows, as it does in the sum over the units
        }
        const float sh = (float)slope, ih = (float)icept;
        if (e_raw < E && (rep == 0 || j == 0))
            val[s] = make_float4(sh, isfinite(sh) ? (float)(slope - sh) : 0.f, ih, isfinite(ih) ? (float)(icept - ih) : 0.f);
    }
}

__device__ __forceinline__ XTable load_table(float* sm, const float* __restrict__ table, int E) {
    for (int i = threadIdx.x; i < (int)x_table_floats(E); i += XTHREADS) sm[i] = table[i];
    return XTable{reinterpret_cast<const float4*>(sm), sm + 4 * E * XSEG};
}

__device__ __forceinline__ float expert_eval(const XTable& p, int e, float g) {
    const float* t = p.t + e * XSEG;
    int s = g > t[7] ? 8 : 0;
    s += g > t[s + 3] ? 4 : 0;
    s += g > t[s + 1] ? 2 : 0;
    s += g > t[s] ? 1 : 0;
    s += g > t[s] ? 1 : 0;
    const float4 v = p.v[e * XSEG + s];
    const float m = __fmul_rn(v.x, g), me = fmaf(v.x, g, -m);                       // m + me = slope * g
    const float q = __fadd_rn(m, v.z), w = __fsub_rn(q, m);
    const float qe = __fadd_rn(__fsub_rn(m, __fsub_rn(q, w)), __fsub_rn(v.z, w));    // q + qe = m + intercept
    const float r = q + ((me + qe) + fmaf(v.y, g, v.w));
    return r == r ? r : fmaf(v.x, g, v.z);                                          // past the range of floats: no inf - inf of the error terms
}

__device__ __forceinline__ int expert_of(int a, int b, int pk, int E) {
    const int e = a * pk + b;
    return e < 0 ? 0 : (e >= E ? E - 1 : e);
}

// one thread per (element, head); the heads of an element are added in head order by the thread of head 0
__global__ void __launch_bounds__(XTHREADS) routed_experts_fwd_kernel(const float* __restrict__ g, const int4* __restrict__ ia,
                                                                      const int4* __restrict__ ib, const float4* __restrict__ wa,
                                                                      const float4* __restrict__ wb, const float* __restrict__ table,
                                                                      int64_t n, int heads, int E, int pk, float* __restrict__ total) {
    extern __shared__ __align__(16) float sm[];
    const XTable p = load_table(sm, table, E);
    float* s_tot = sm + x_table_floats(E);
    __syncthreads();
    const int epc = XTHREADS / heads;                                   // elements per CTA
    const int le = threadIdx.x / heads, h = threadIdx.x % heads;
    const int64_t elem = (int64_t)blockIdx.x * epc + le;
    float t = 0.f;
    if (le < epc && elem < n) {
        const float gv = g[elem];
        const int64_t r = elem * heads + h;
        const int4 a4 = ia[r], b4 = ib[r];
        const float4 wa4 = wa[r], wb4 = wb[r];
        const int av[XK] = {a4.x, a4.y, a4.z, a4.w}, bv[XK] = {b4.x, b4.y, b4.z, b4.w};
        const float wav[XK] = {wa4.x, wa4.y, wa4.z, wa4.w}, wbv[XK] = {wb4.x, wb4.y, wb4.z, wb4.w};
#pragma unroll
        for (int a = 0; a < XK; ++a)
#pragma unroll
            for (int b = 0; b < XK; ++b) {
                t = fmaf(wav[a] * wbv[b], expert_eval(p, expert_of(av[a], bv[b], pk, E), gv), t);
            }
    }
    s_tot[threadIdx.x] = t;
    __syncthreads();
    if (h == 0 && le < epc && elem < n) {
        float s = 0.f;
        for (int k = 0; k < heads; ++k) s += s_tot[threadIdx.x + k];
        total[elem] = s;
    }
}

// Persistent CTAs over tiles of XTHREADS / heads elements.  partial: [gridDim.x, 3*E*XH + E] (dW1, db1, dW2, db2).
__global__ void __launch_bounds__(XTHREADS, 2) routed_experts_bwd_kernel(const float* __restrict__ g, const int4* __restrict__ ia,
                                                                      const int4* __restrict__ ib, const float4* __restrict__ wa,
                                                                      const float4* __restrict__ wb, const float* __restrict__ W1,
                                                                      const float* __restrict__ b1, const float* __restrict__ W2,
                                                                      const float* __restrict__ table, const float* __restrict__ dtotal,
                                                                      int64_t n, int heads, int E, int pk, float4* __restrict__ dwa,
                                                                      float4* __restrict__ dwb, float* __restrict__ partial) {
    extern __shared__ __align__(16) float sm[];
    const XTable p = load_table(sm, table, E);
    const int epc = XTHREADS / heads;
    float* s_g = sm + x_table_floats(E);                                // [epc]
    float* s_route = s_g + XTHREADS;                                    // [epc][XE]
    __syncthreads();
    const int le = threadIdx.x / heads, h = threadIdx.x % heads;
    // the (expert, hidden unit) pairs of this thread: hidden unit j is fixed, experts e0 + 16 q
    const int j = threadIdx.x & (XH - 1), e0 = threadIdx.x / XH;
    // per pair: sums of c * g, c and c * z over the elements whose unit is on (c: the element's routing weight times its gradient)
    float w1r[XMAXQ], b1r[XMAXQ], cg[XMAXQ], c0[XMAXQ], cz[XMAXQ], csum = 0.f;
#pragma unroll
    for (int q = 0; q < XMAXQ; ++q) {
        const int e = e0 + (XTHREADS / XH) * q;
        const bool in = e < E;
        w1r[q] = in ? W1[e * XH + j] : 0.f;
        b1r[q] = in ? b1[e * XH + j] : 0.f;
        cg[q] = c0[q] = cz[q] = 0.f;
    }
    const int64_t tiles = (n + epc - 1) / epc;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t elem = tile * epc + le;
        const bool live = le < epc && elem < n;
        int av[XK] = {0, 0, 0, 0}, bv[XK] = {0, 0, 0, 0};
        float wav[XK], wbv[XK], dt = 0.f;
        if (live) {
            const float gv = g[elem];
            dt = dtotal[elem];
            const int64_t r = elem * heads + h;
            const int4 a4 = ia[r], b4 = ib[r];
            const float4 wa4 = wa[r], wb4 = wb[r];
            av[0] = a4.x; av[1] = a4.y; av[2] = a4.z; av[3] = a4.w; bv[0] = b4.x; bv[1] = b4.y; bv[2] = b4.z; bv[3] = b4.w;
            wav[0] = wa4.x; wav[1] = wa4.y; wav[2] = wa4.z; wav[3] = wa4.w; wbv[0] = wb4.x; wbv[1] = wb4.y; wbv[2] = wb4.z; wbv[3] = wb4.w;
            float da[XK] = {0.f, 0.f, 0.f, 0.f}, db[XK] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int a = 0; a < XK; ++a)
#pragma unroll
                for (int b = 0; b < XK; ++b) {
                    const float dw = dt * expert_eval(p, expert_of(av[a], bv[b], pk, E), gv);       // d total / d (wa*wb) times the incoming gradient
                    da[a] = fmaf(dw, wbv[b], da[a]);
                    db[b] = fmaf(dw, wav[a], db[b]);
                }
            dwa[r] = make_float4(da[0], da[1], da[2], da[3]);
            dwb[r] = make_float4(db[0], db[1], db[2], db[3]);
            if (h == 0) s_g[le] = gv;
        } else if (h == 0 && le < epc) {
            s_g[le] = 0.f;
        }
        for (int i = threadIdx.x; i < epc * XE; i += XTHREADS) s_route[i] = 0.f;
        __syncthreads();
        // head after head: within one head the 16 experts of an element are distinct when its keys are (top-k indices are);
        // repeated keys would still be added by one thread, in a fixed order
        for (int hh = 0; hh < heads; ++hh) {
            if (live && h == hh) {
#pragma unroll
                for (int k = 0; k < XK * XK; ++k) s_route[le * XE + expert_of(av[k / XK], bv[k % XK], pk, E)] += dt * wav[k / XK] * wbv[k % XK];
            }
            __syncthreads();
        }
        const int64_t left = n - tile * epc;
        const int cnt = left < epc ? (int)left : epc;
        for (int m = 0; m < cnt; ++m) {
            const float gm = s_g[m];
            const float* rt = s_route + m * XE + e0;
#pragma unroll
            for (int q = 0; q < XMAXQ; ++q) {                         // without branches: about half of the entries are zero, but never a whole warp's
                const float z = fmaf(gm, w1r[q], b1r[q]);
                const float c = z > 0.f ? rt[(XTHREADS / XH) * q] : 0.f;
                cz[q] = fmaf(c, z, cz[q]); cg[q] = fmaf(c, gm, cg[q]); c0[q] += c;
            }
        }
        if (threadIdx.x < E)
            for (int m = 0; m < cnt; ++m) csum += s_route[m * XE + threadIdx.x];
        __syncthreads();                                               // the tables are rewritten by the next tile
    }
    float* out = partial + (int64_t)blockIdx.x * (3 * E * XH + E);
#pragma unroll
    for (int q = 0; q < XMAXQ; ++q) {
        const int e = e0 + (XTHREADS / XH) * q;
        if (e < E) {
            const float w2 = W2[e * XH + j];
            out[e * XH + j] = w2 * cg[q];
            out[E * XH + e * XH + j] = w2 * c0[q];
            out[2 * E * XH + e * XH + j] = cz[q];
        }
    }
    if (threadIdx.x < E) out[3 * E * XH + threadIdx.x] = csum;
}

size_t fwd_smem(int E) { return (size_t)(x_table_floats(E) + XTHREADS) * sizeof(float); }
size_t bwd_smem(int E, int heads) { return (size_t)(x_table_floats(E) + XTHREADS + (XTHREADS / heads) * XE) * sizeof(float); }

}  // namespace

bool routed_experts_supported(int heads, int E, int hidden, int topk) {
    return hidden == XH && topk == XK && heads >= 1 && heads <= 16 && E >= 1 && E <= (XTHREADS / XH) * XMAXQ && bwd_smem(E, heads) <= 200 * 1024;
}

// CTAs of the backward pass = rows of `partial` ([ctas, 3*E*16 + E] floats)
int routed_experts_bwd_ctas(int64_t n, int heads) {
    const int epc = XTHREADS / heads;
    const int64_t tiles = (n + epc - 1) / epc;
    const int64_t cap = 2 * 148;
    return (int)(tiles < cap ? (tiles < 1 ? 1 : tiles) : cap);
}

// floats of scratch for the value tables of E experts
int routed_experts_table_floats(int E) { return (int)x_table_floats(E); }

int routed_experts_fwd(const float* g, const int* ia, const int* ib, const float* wa, const float* wb, const float* W1, const float* b1,
                       const float* W2, const float* b2, int64_t n, int heads, int E, int pk, float* table, float* total, cudaStream_t s) {
    if (n <= 0) return 0;
    const size_t smem = fwd_smem(E);
    if (cudaFuncSetAttribute(routed_experts_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 2;
    const int epc = XTHREADS / heads;
    count_launch(2);
    experts_table_kernel<<<(E + 7) / 8, 128, 0, s>>>(W1, b1, W2, b2, E, table);
    routed_experts_fwd_kernel<<<(unsigned)((n + epc - 1) / epc), XTHREADS, smem, s>>>(
        g, (const int4*)ia, (const int4*)ib, (const float4*)wa, (const float4*)wb, table, n, heads, E, pk, total);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

int routed_experts_bwd(const float* g, const int* ia, const int* ib, const float* wa, const float* wb, const float* W1, const float* b1,
                       const float* W2, const float* b2, const float* dtotal, int64_t n, int heads, int E, int pk, float* dwa, float* dwb,
                       float* table, float* partial, float* dparams, cudaStream_t s) {
    const int ng = 3 * E * XH + E;
    if (n <= 0) return cudaMemsetAsync(dparams, 0, (size_t)ng * sizeof(float), s) == cudaSuccess ? 0 : 3;
    const size_t smem = bwd_smem(E, heads);
    if (cudaFuncSetAttribute(routed_experts_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 2;
    const int ctas = routed_experts_bwd_ctas(n, heads);
    count_launch(3);
    experts_table_kernel<<<(E + 7) / 8, 128, 0, s>>>(W1, b1, W2, b2, E, table);
    routed_experts_bwd_kernel<<<ctas, XTHREADS, smem, s>>>(g, (const int4*)ia, (const int4*)ib, (const float4*)wa, (const float4*)wb, W1, b1, W2,
                                                          table, dtotal, n, heads, E, pk, (float4*)dwa, (float4*)dwb, partial);
    column_parts_kernel<<<(ng + 31) / 32, 1024, 0, s>>>(partial, ctas, ng, dparams);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace sg
