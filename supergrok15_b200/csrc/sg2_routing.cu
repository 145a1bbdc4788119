// Product-key routing of the SuperGrok v2 bilevel path as two kernels (sm_100a); the arithmetic is csrc/sg2_routing_math.h.
//
// Forward: one thread per (element, head): query, 2 x pk scores, top-4 and softmax per sub-key; writes ia, ib, wa, wb [n, heads, 4]
// (the inputs of the routed expert kernels, csrc/sg2_experts.cu).  Backward: the same thread recomputes its query, turns d wa / d wb
// into score and query gradients, and the tile's query gradients are folded back through Wq into d pin [n, P]; the parameter
// gradients (Wq, both key tables) are summed without atomics: every thread owns fixed outputs, walks the tile's elements in
// shared memory, keeps its sums in registers across tiles and writes them once per CTA; a second kernel adds the CTAs in order.
// It replaces two matrix products, a block-diagonal assembly, a top-k and a softmax over [n, 2 * heads * pk] tensors (and their
// autograd graph) of the PyTorch statement in optim/metanet.py: soft_head.
#include "sg_native.h"
#include "sg2_routing_math.h"
#include "column_parts.cuh"

namespace sg {
namespace {
using namespace routing;

constexpr int RT = 256;                   // threads per CTA
constexpr int RMAXW = 4;                  // Wq outputs per thread (heads * 8 * P <= 1024)
constexpr int RMAXK = 2;                  // key-table outputs per thread (2 * heads * pk * 4 <= 512)

struct RWeights { const float* wq; const float* ka; const float* kb; };

__device__ __forceinline__ RWeights stage_weights(float* sm, const float* __restrict__ Wq, const float* __restrict__ KA,
                                                  const float* __restrict__ KB, int heads, int P, int pk) {
    float* wq = sm;
    float* ka = wq + heads * RD * P;
    float* kb = ka + heads * pk * RH;
    for (int i = threadIdx.x; i < heads * RD * P; i += RT) wq[i] = Wq[i];
    for (int i = threadIdx.x; i < heads * pk * RH; i += RT) { ka[i] = KA[i]; kb[i] = KB[i]; }
    return RWeights{wq, ka, kb};
}
__host__ __device__ inline int weights_floats(int heads, int P, int pk) { return heads * RD * P + 2 * heads * pk * RH; }

// CP / CPK > 0: input width and key rows are compile-time constants (loops unroll, the per-element arrays stay in registers)
template <int CP, int CPK>
__global__ void __launch_bounds__(RT) routing_fwd_kernel(const float* __restrict__ pin, const float* __restrict__ Wq, const float* __restrict__ KA,
                                                         const float* __restrict__ KB, int64_t n, int heads, int P_rt, int pk_rt,
                                                         int4* __restrict__ ia, int4* __restrict__ ib, float4* __restrict__ wa,
                                                         float4* __restrict__ wb) {
    const int P = CP > 0 ? CP : P_rt, pk = CPK > 0 ? CPK : pk_rt;
    extern __shared__ float sm[];
    const RWeights w = stage_weights(sm, Wq, KA, KB, heads, P, pk);
    __syncthreads();
    const int epc = RT / heads;
    const int le = threadIdx.x / heads, h = threadIdx.x % heads;
    const int64_t elem = (int64_t)blockIdx.x * epc + le;
    if (le >= epc || elem >= n) return;
    float x[CP > 0 ? CP : RP_MAX], q[RD], a_w[RK], b_w[RK];
    int a_i[RK], b_i[RK];
#pragma unroll
    for (int j = 0; j < P; ++j) x[j] = pin[elem * P + j];
    route_fwd(x, P, w.wq + h * RD * P, w.ka + h * pk * RH, w.kb + h * pk * RH, pk, q, a_i, b_i, a_w, b_w);
    const int64_t r = elem * heads + h;
    ia[r] = make_int4(a_i[0], a_i[1], a_i[2], a_i[3]);
    ib[r] = make_int4(b_i[0], b_i[1], b_i[2], b_i[3]);
    wa[r] = make_float4(a_w[0], a_w[1], a_w[2], a_w[3]);
    wb[r] = make_float4(b_w[0], b_w[1], b_w[2], b_w[3]);
}

// partial: [gridDim.x, heads*8*P + 2*heads*pk*4]  (d Wq | d KA | d KB)
__global__ void __launch_bounds__(RT) routing_bwd_kernel(const float* __restrict__ pin, const float* __restrict__ Wq, const float* __restrict__ KA,
                                                         const float* __restrict__ KB, const int4* __restrict__ ia, const int4* __restrict__ ib,
                                                         const float4* __restrict__ wa, const float4* __restrict__ wb,
                                                         const float4* __restrict__ dwa, const float4* __restrict__ dwb, int64_t n, int heads,
                                                         int P, int pk, float* __restrict__ dpin, float* __restrict__ partial) {
    extern __shared__ float sm[];
    const RWeights w = stage_weights(sm, Wq, KA, KB, heads, P, pk);
    const int epc = RT / heads;
    float* s_pin = sm + weights_floats(heads, P, pk);              // [epc][P]
    float* s_q = s_pin + epc * P;                                  // [epc][heads][8]
    float* s_dq = s_q + epc * heads * RD;                          // [epc][heads][8]
    float* s_dt = s_dq + epc * heads * RD;                         // [epc][heads][8]   (A scores 0..3, B scores 4..7)
    int* s_ix = reinterpret_cast<int*>(s_dt + epc * heads * RD);   // [epc][heads][8]
    const int le = threadIdx.x / heads, h = threadIdx.x % heads;
    const int n_wq = heads * RD * P, n_k = heads * pk * RH;
    float acc_w[RMAXW], acc_k[RMAXK];
#pragma unroll
    for (int u = 0; u < RMAXW; ++u) acc_w[u] = 0.f;
#pragma unroll
    for (int u = 0; u < RMAXK; ++u) acc_k[u] = 0.f;
    __syncthreads();
    const int64_t tiles = (n + epc - 1) / epc;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t left = n - tile * epc;
        const int cnt = left < epc ? (int)left : epc;
        for (int i = threadIdx.x; i < cnt * P; i += RT) s_pin[i] = pin[tile * epc * P + i];
        __syncthreads();
        const bool live = le < cnt;
        if (live) {
            const int64_t r = (tile * epc + le) * heads + h;
            const int4 a4 = ia[r], b4 = ib[r];
            const float4 wa4 = wa[r], wb4 = wb[r], da4 = dwa[r], db4 = dwb[r];
            const int a_i[RK] = {a4.x, a4.y, a4.z, a4.w}, b_i[RK] = {b4.x, b4.y, b4.z, b4.w};
            const float a_w[RK] = {wa4.x, wa4.y, wa4.z, wa4.w}, b_w[RK] = {wb4.x, wb4.y, wb4.z, wb4.w};
            const float a_d[RK] = {da4.x, da4.y, da4.z, da4.w}, b_d[RK] = {db4.x, db4.y, db4.z, db4.w};
            float q[RD], dt[2 * RK], dq[RD];
            query(s_pin + le * P, P, w.wq + h * RD * P, q);
            route_bwd(a_i, b_i, a_w, b_w, a_d, b_d, w.ka + h * pk * RH, w.kb + h * pk * RH, dt, dq);
            const int o = (le * heads + h) * RD;
#pragma unroll
            for (int k = 0; k < RD; ++k) { s_q[o + k] = q[k]; s_dq[o + k] = dq[k]; s_dt[o + k] = dt[k]; }
#pragma unroll
            for (int k = 0; k < RK; ++k) { s_ix[o + k] = a_i[k]; s_ix[o + RK + k] = b_i[k]; }
        }
        __syncthreads();
        if (live) {                                               // d pin[j] = sum over heads and query rows of Wq[hh][o][j] * dq[hh][o]
            const float* dqe = s_dq + le * heads * RD;
            for (int j = h; j < P; j += heads) {
                float a = 0.f;
                for (int t = 0; t < heads * RD; ++t) a = fmaf(w.wq[t * P + j], dqe[t], a);
                dpin[(tile * epc + le) * P + j] = a;
            }
        }
        // parameter gradients: fixed outputs per thread, elements of the tile in order
#pragma unroll
        for (int u = 0; u < RMAXW; ++u) {
            const int id = threadIdx.x + u * RT;
            if (id < n_wq) {
                const int row = id / P, j = id % P;               // row = head * 8 + query row
                float a = acc_w[u];
                for (int m = 0; m < cnt; ++m) a = fmaf(s_dq[m * heads * RD + row], s_pin[m * P + j], a);
                acc_w[u] = a;
            }
        }
#pragma unroll
        for (int u = 0; u < RMAXK; ++u) {
            const int id = threadIdx.x + u * RT;
            if (id < 2 * n_k) {
                const int ab = id / n_k, rem = id % n_k;          // ab: 0 = table A, 1 = table B
                const int hh = rem / (pk * RH), row = (rem / RH) % pk, d = rem % RH;
                float a = acc_k[u];
                for (int m = 0; m < cnt; ++m) {
                    const int o = (m * heads + hh) * RD + ab * RK;
#pragma unroll
                    for (int k = 0; k < RK; ++k)
                        if (s_ix[o + k] == row) a = fmaf(s_dt[o + k], s_q[(m * heads + hh) * RD + ab * RH + d], a);
                }
                acc_k[u] = a;
            }
        }
        __syncthreads();                                          // the tile buffers are rewritten next
    }
    float* out = partial + (int64_t)blockIdx.x * (n_wq + 2 * n_k);
#pragma unroll
    for (int u = 0; u < RMAXW; ++u) { const int id = threadIdx.x + u * RT; if (id < n_wq) out[id] = acc_w[u]; }
#pragma unroll
    for (int u = 0; u < RMAXK; ++u) { const int id = threadIdx.x + u * RT; if (id < 2 * n_k) out[n_wq + id] = acc_k[u]; }
}

// The same for the default meta-net (4 heads, 22 inputs, 12 key rows), with the operands of every product in registers.  A thread of
// (element, head) reads a row of Wq once, as six 16-byte loads, for both the query and d pin; the heads' d pin meet by shuffles.  The parameter
// gradients are outer products summed over the tile: a warp takes every eighth element, a lane a 4 x 6 block of d Wq and a 3 x 4 block
// of one key table (whose score gradients stand in a dense row of 12), so that five loads feed 36 FMAs; the eight warps are added in order
// at the end.  Bound by instruction issue; 422,755 elements: 818 -> 147 us (two shared-memory loads per FMA before).
namespace fixed {
constexpr int H = 4, P = 22, PP = 24, PK = 12, TILE = RT / H;
constexpr int WHEAD = 8 * PP + 4;                              // row pitch 24, heads 4 floats apart in the banks
constexpr int QP = 36, SP = 100;                                // pitches of [32] query rows and [96] dense score gradients: odd in float4
constexpr int N_WQ = H * 8 * P, N_K = H * PK * 4, NG = N_WQ + 2 * N_K;
constexpr int F_W = 0, F_K = F_W + H * WHEAD, F_X = F_K + 2 * N_K, F_Q = F_X + TILE * PP, F_DQ = F_Q + TILE * QP, F_DS = F_DQ + TILE * QP,
              FLOATS = F_DS + TILE * SP;
static_assert(8 * NG <= FLOATS - F_X, "the warps' sums fit where the tile was");
}  // namespace fixed

__global__ void __launch_bounds__(RT, 2) routing_bwd_default_kernel(const float* __restrict__ pin, const float* __restrict__ Wq, const float* __restrict__ KA,
                                                                    const float* __restrict__ KB, const int4* __restrict__ ia, const int4* __restrict__ ib,
                                                                    const float4* __restrict__ wa, const float4* __restrict__ wb,
                                                                    const float4* __restrict__ dwa, const float4* __restrict__ dwb, int64_t n,
                                                                    float* __restrict__ dpin, float* __restrict__ partial) {
    using namespace fixed;
    extern __shared__ __align__(16) float sm[];
    float *s_w = sm + F_W, *s_k = sm + F_K, *s_x = sm + F_X, *s_q = sm + F_Q, *s_dq = sm + F_DQ, *s_ds = sm + F_DS;
    for (int i = threadIdx.x; i < H * 8 * PP; i += RT) {
        const int r = i / PP, j = i % PP;
        s_w[(r / 8) * WHEAD + (r % 8) * PP + j] = j < P ? Wq[r * P + j] : 0.f;
    }
    for (int i = threadIdx.x; i < N_K; i += RT) { s_k[i] = KA[i]; s_k[N_K + i] = KB[i]; }
    for (int i = threadIdx.x; i < TILE * (PP - P); i += RT) s_x[(i / (PP - P)) * PP + P + i % (PP - P)] = 0.f;
    const int le = threadIdx.x / H, h = threadIdx.x % H, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rg = lane >> 2, cg = lane & 3;                    // d Wq rows 4 rg .. + 3, columns 6 cg .. + 5; key table rg & 1 of head rg >> 1, rows 3 cg .. + 2
    float aw[4][6], ak[3][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 6; ++v) aw[u][v] = 0.f;
#pragma unroll
    for (int u = 0; u < 3; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) ak[u][v] = 0.f;
    const int64_t tiles = (n + TILE - 1) / TILE;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t left = n - tile * TILE;
        const int cnt = left < TILE ? (int)left : TILE;
        __syncthreads();                                        // the previous tile's sums have been taken
        for (int i = threadIdx.x; i < cnt * P; i += RT) s_x[(i / P) * PP + i % P] = pin[tile * TILE * P + i];
        __syncthreads();
        const bool live = le < cnt;
        float dt[8], dq[8], q[8], dp[PP];
#pragma unroll
        for (int k = 0; k < 8; ++k) dq[k] = 0.f;
#pragma unroll
        for (int j = 0; j < PP; ++j) dp[j] = 0.f;
        if (live) {
            const int64_t r = (tile * TILE + le) * H + h;
            const int4 a4 = ia[r], b4 = ib[r];
            const float4 wa4 = wa[r], wb4 = wb[r], da4 = dwa[r], db4 = dwb[r];
            const int a_i[RK] = {a4.x, a4.y, a4.z, a4.w}, b_i[RK] = {b4.x, b4.y, b4.z, b4.w};
            const float a_w[RK] = {wa4.x, wa4.y, wa4.z, wa4.w}, b_w[RK] = {wb4.x, wb4.y, wb4.z, wb4.w};
            const float a_d[RK] = {da4.x, da4.y, da4.z, da4.w}, b_d[RK] = {db4.x, db4.y, db4.z, db4.w};
            route_bwd(a_i, b_i, a_w, b_w, a_d, b_d, s_k + h * PK * RH, s_k + N_K + h * PK * RH, dt, dq);
            float4* ds = reinterpret_cast<float4*>(s_ds + le * SP + h * 2 * PK);
#pragma unroll
            for (int k = 0; k < 6; ++k) ds[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            float* dsf = s_ds + le * SP + h * 2 * PK;
#pragma unroll
            for (int k = 0; k < RK; ++k) { dsf[a_i[k]] += dt[k]; dsf[PK + b_i[k]] += dt[RK + k]; }
            float x[PP];
#pragma unroll
            for (int j = 0; j < PP / 4; ++j) {
                const float4 v = reinterpret_cast<const float4*>(s_x + le * PP)[j];
                x[4 * j] = v.x; x[4 * j + 1] = v.y; x[4 * j + 2] = v.z; x[4 * j + 3] = v.w;
            }
#pragma unroll
            for (int o = 0; o < 8; ++o) {
                float acc = 0.f;
#pragma unroll
                for (int j = 0; j < PP / 4; ++j) {
                    const float4 v = reinterpret_cast<const float4*>(s_w + h * WHEAD + o * PP)[j];
                    acc = fmaf(v.x, x[4 * j], acc); acc = fmaf(v.y, x[4 * j + 1], acc); acc = fmaf(v.z, x[4 * j + 2], acc); acc = fmaf(v.w, x[4 * j + 3], acc);
                    dp[4 * j] = fmaf(v.x, dq[o], dp[4 * j]); dp[4 * j + 1] = fmaf(v.y, dq[o], dp[4 * j + 1]);
                    dp[4 * j + 2] = fmaf(v.z, dq[o], dp[4 * j + 2]); dp[4 * j + 3] = fmaf(v.w, dq[o], dp[4 * j + 3]);
                }
                q[o] = acc;
            }
            float4* qo = reinterpret_cast<float4*>(s_q + le * QP + h * 8);
            qo[0] = make_float4(q[0], q[1], q[2], q[3]); qo[1] = make_float4(q[4], q[5], q[6], q[7]);
            float4* dqo = reinterpret_cast<float4*>(s_dq + le * QP + h * 8);
            dqo[0] = make_float4(dq[0], dq[1], dq[2], dq[3]); dqo[1] = make_float4(dq[4], dq[5], dq[6], dq[7]);
        }
        {   // sum of d pin over the four heads (four neighbouring lanes); each keeps six columns
            const bool hi = (h & 2) != 0, odd = (h & 1) != 0;
            float a[12], c[6];
#pragma unroll
            for (int j = 0; j < 12; ++j) {
                const float got = __shfl_xor_sync(0xffffffffu, hi ? dp[j] : dp[12 + j], 2);
                a[j] = (hi ? dp[12 + j] : dp[j]) + got;
            }
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const float got = __shfl_xor_sync(0xffffffffu, odd ? a[j] : a[6 + j], 1);
                c[j] = (odd ? a[6 + j] : a[j]) + got;
            }
            const int base = (hi ? 12 : 0) + (odd ? 6 : 0);
            if (live)
#pragma unroll
                for (int j = 0; j < 6; ++j)
                    if (base + j < P) dpin[(tile * TILE + le) * P + base + j] = c[j];
        }
        __syncthreads();
        for (int m = warp; m < cnt; m += RT / 32) {
            const float4 d = *reinterpret_cast<const float4*>(s_dq + m * QP + 4 * rg), qv = *reinterpret_cast<const float4*>(s_q + m * QP + 4 * rg);
            float x[6];
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                const float2 t = reinterpret_cast<const float2*>(s_x + m * PP + 6 * cg)[v];
                x[2 * v] = t.x; x[2 * v + 1] = t.y;
            }
            const float dr[4] = {d.x, d.y, d.z, d.w}, qr[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 6; ++v) aw[u][v] = fmaf(dr[u], x[v], aw[u][v]);
            const float* ds = s_ds + m * SP + rg * PK + 3 * cg;   // [head][A, B][12]: rg = 2 head + table
#pragma unroll
            for (int u = 0; u < 3; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) ak[u][v] = fmaf(ds[u], qr[v], ak[u][v]);
        }
    }
    __syncthreads();
    float* red = s_x + warp * NG;
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 6; ++v)
            if (6 * cg + v < P) red[(4 * rg + u) * P + 6 * cg + v] = aw[u][v];
#pragma unroll
    for (int u = 0; u < 3; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) red[N_WQ + (rg & 1) * N_K + ((rg >> 1) * PK + 3 * cg + u) * 4 + v] = ak[u][v];
    __syncthreads();
    for (int i = threadIdx.x; i < NG; i += RT) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < RT / 32; ++w) t += s_x[w * NG + i];
        partial[(int64_t)blockIdx.x * NG + i] = t;
    }
}

size_t fwd_smem(int heads, int P, int pk) { return (size_t)weights_floats(heads, P, pk) * sizeof(float); }
size_t bwd_smem(int heads, int P, int pk) {
    const int epc = RT / heads;
    return (size_t)(weights_floats(heads, P, pk) + epc * P + 4 * epc * heads * RD) * sizeof(float);
}
}  // namespace

bool routing_supported(int heads, int P, int pk, int d_model, int topk) {
    return d_model == routing::RD && topk == routing::RK && heads >= 1 && heads <= 16 && P >= 1 && P <= routing::RP_MAX && pk >= routing::RK &&
           pk <= routing::RPK_MAX && heads * routing::RD * P <= RMAXW * RT && 2 * heads * pk * routing::RH <= RMAXK * RT &&
           bwd_smem(heads, P, pk) <= 200 * 1024;
}
int routing_bwd_ctas(int64_t n, int heads) {
    const int epc = RT / heads;
    const int64_t tiles = (n + epc - 1) / epc;
    return (int)(tiles < 1 ? 1 : (tiles < 4 * 148 ? tiles : 4 * 148));
}
int routing_ng(int heads, int P, int pk) { return heads * routing::RD * P + 2 * heads * pk * routing::RH; }

int routing_fwd(const float* pin, const float* Wq, const float* KA, const float* KB, int64_t n, int heads, int P, int pk, int* ia, int* ib,
                float* wa, float* wb, cudaStream_t s) {
    if (n <= 0) return 0;
    const size_t smem = fwd_smem(heads, P, pk);
    if (cudaFuncSetAttribute(routing_fwd_kernel<22, 12>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaFuncSetAttribute(routing_fwd_kernel<0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 2;
    const int epc = RT / heads;
    const unsigned grid = (unsigned)((n + epc - 1) / epc);
    count_launch();
    if (P == 22 && pk == 12)                                          // the default meta-net: gru 4 + 2 * d_model 16 + 2 inputs, 144 experts
        routing_fwd_kernel<22, 12><<<grid, RT, smem, s>>>(pin, Wq, KA, KB, n, heads, P, pk, (int4*)ia, (int4*)ib, (float4*)wa, (float4*)wb);
    else
        routing_fwd_kernel<0, 0><<<grid, RT, smem, s>>>(pin, Wq, KA, KB, n, heads, P, pk, (int4*)ia, (int4*)ib, (float4*)wa, (float4*)wb);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

int routing_bwd(const float* pin, const float* Wq, const float* KA, const float* KB, const int* ia, const int* ib, const float* wa, const float* wb,
                const float* dwa, const float* dwb, int64_t n, int heads, int P, int pk, float* dpin, float* partial, float* dparams, cudaStream_t s) {
    const int ng = routing_ng(heads, P, pk);
    if (n <= 0) return cudaMemsetAsync(dparams, 0, (size_t)ng * sizeof(float), s) == cudaSuccess ? 0 : 3;
    const size_t smem = bwd_smem(heads, P, pk);
    if (cudaFuncSetAttribute(routing_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 2;
    int ctas = routing_bwd_ctas(n, heads);
    count_launch(2);
    if (heads == fixed::H && P == fixed::P && pk == fixed::PK) {
        const size_t fsm = (size_t)fixed::FLOATS * sizeof(float);
        if (cudaFuncSetAttribute(routing_bwd_default_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fsm) != cudaSuccess) return 2;
        ctas = ctas < 2 * 148 ? ctas : 2 * 148;
        routing_bwd_default_kernel<<<ctas, RT, fsm, s>>>(pin, Wq, KA, KB, (const int4*)ia, (const int4*)ib, (const float4*)wa, (const float4*)wb,
                                                         (const float4*)dwa, (const float4*)dwb, n, dpin, partial);
    } else
        routing_bwd_kernel<<<ctas, RT, smem, s>>>(pin, Wq, KA, KB, (const int4*)ia, (const int4*)ib, (const float4*)wa, (const float4*)wb,
                                                  (const float4*)dwa, (const float4*)dwb, n, heads, P, pk, dpin, partial);
    column_parts_kernel<<<(ng + 31) / 32, 1024, 0, s>>>(partial, ctas, ng, dparams);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace sg
