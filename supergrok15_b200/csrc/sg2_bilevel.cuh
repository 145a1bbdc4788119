// Adjoint of the bidirectional Mamba-3 scan (bilevel meta-learning path), included at the end of sg2_kernels.cu so it
// shares the __constant__ weight block of that translation unit.
//
// The reference runs this adjoint serially: one 16-thread CTA per parameter tensor walks N timesteps backwards
// (csrc/supergrok2_mamba_peer_backward_kernels.cu:1043, :1506) and drops the cross-column terms of d_x.  Here the adjoint
// uses the same chunk decomposition as the forward scan, so every SM works on it:
//
//   adj 1   per chunk: aggregate of the reverse recurrence  dh[t-1] = M_t^T (dh[t] + dy_t C_t)   (prefix product walked
//           forwards from the chunk start, with an early exit at 2^-100; the forward aggregates stop at 2^-48)
//   adj 2   carry: dh arriving at the end of every chunk (chunks in reverse order; the last chunk receives zero)
//   adj 3   per chunk: walk the tiles backwards from the states that the forward scan has left at their boundaries (global scratch):
//           recompute the 16 states of the tile into shared memory, run the exact adjoint of each timestep, accumulate parameter
//           gradients privately per lane
//   adj 4   fixed-order reduction of the per-item partial gradients
//
// Because x, z, dt, B and C are affine in (g, s) (SG2Pack::AFF* tables), their weight gradients are gradients of the
// TABLES:  dU[j][k] += d value_j[t] * (g_t, s_t, 1)[k].  The chain rule from the tables to input_proj / in_proj / dt_proj /
// B_proj / C_proj is a handful of tiny matrix products (sg2_meta.cu: sg2_fold_bwd_kernel).  This formulation contains the
// cross-column terms exactly (every column's dependence on B_s and C_s goes through the shared tables).
// Per direction the kernels produce BL_NG = 768 gradient values:
//   [0,256)    d A_log [16][16]          [256,384)  d rope_freq [16][8]      [384,400)  d D [16]
//   [400,448)  d U_x [16][3]   [448,496) d U_z   [496,544) d U_dt   [544,592) d U_B [16][3]   [592,640) d U_C [16][3]
//   [640,768)  d out_proj [8][16]
#pragma once

namespace sg {
namespace {

constexpr int BL_TILE = 16;                    // timesteps per backward tile
constexpr int BL_ITEMS = 4;                    // items per CTA of adj 1
constexpr int BL_THREADS = BL_ITEMS * 16;
constexpr int BL_NG = 768;                     // gradient values per direction (layout above)
constexpr int BL_ROW = 60;                     // floats per timestep row in shared memory: B16 C16 (g,s,-,-) gout16 dctx8

// g_out_j[t] = sum_d dctx[t][d] * Wout[d][j]  and  B, C of the timestep: lane l = timestep
template <int DIR>
__device__ __forceinline__ void bl_stage_a(float* __restrict__ tile, const float2* __restrict__ gs, const uint32_t* __restrict__ vals_sorted,
                                           const float* __restrict__ dctx, int64_t off, int n, int u, bool valid, int l) {
    constexpr int W = (DIR == 0) ? P::DIR0 : P::DIR1;
    constexpr int AF = (DIR == 0) ? P::AFF0 : P::AFF1;
    if (!valid) return;
    float4* row = reinterpret_cast<float4*>(tile + l * BL_ROW);
    const int pos = (DIR == 0) ? u : (n - 1 - u);
    const float2 v = gs[off + pos];
    float bc[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const int w = AF + P::A_B + 3 * k;
        bc[k] = fmaf(c_w[w], v.x, fmaf(c_w[w + 1], v.y, c_w[w + 2]));
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) row[q] = make_float4(bc[4 * q], bc[4 * q + 2], bc[4 * q + 1], bc[4 * q + 3]);      // order of row_pos()
    row[8] = make_float4(v.x, v.y, 0.f, 0.f);
    const uint32_t orig = vals_sorted[off + pos];
    const float4* dc = reinterpret_cast<const float4*>(dctx + (int64_t)orig * 16 + DIR * 8);
    const float4 d0 = dc[0], d1 = dc[1];
    const float d8[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
    float go[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        float acc = 0.f;
#pragma unroll
        for (int d = 0; d < 8; ++d) acc = fmaf(d8[d], c_w[W + P::D_OUT + d * 16 + j], acc);
        go[j] = acc;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) row[9 + q] = make_float4(go[4 * q], go[4 * q + 1], go[4 * q + 2], go[4 * q + 3]);
    row[13] = d0; row[14] = d1;
}

// ---- adj 1: aggregate of the reverse recurrence over a chunk (walked forwards from the chunk start) ----
template <int DIR>
__device__ void bl_adj1(const Item& it, const float2* __restrict__ gs, const uint32_t* __restrict__ vals_sorted, const float* __restrict__ dctx,
                        float* __restrict__ agg, float* __restrict__ tile, int item_idx, int j, unsigned hmask) {
    ColConst<DIR> cc;
    cc.load(j);
    float acc[16], m[32];                         // P (2x2 per pair) and accumulated injection
#pragma unroll
    for (int s = 0; s < 16; ++s) acc[s] = 0.f;
#pragma unroll
    for (int p = 0; p < 8; ++p) { m[4 * p] = 1.f; m[4 * p + 1] = 0.f; m[4 * p + 2] = 0.f; m[4 * p + 3] = 1.f; }
    for (int u0 = it.ub; u0 < it.ue; u0 += BL_TILE) {
        const int cnt = (it.ue - u0 < BL_TILE) ? (it.ue - u0) : BL_TILE;
        bl_stage_a<DIR>(tile, gs, vals_sorted, dctx, it.off, it.n, u0 + j, j < cnt, j);
        __syncwarp(hmask);
        for (int l = 0; l < cnt; ++l) {
            const float* row = tile + l * BL_ROW;
            const float2 v = *reinterpret_cast<const float2*>(row + 32);
            const float z = fmaf(cc.uz[0], v.x, fmaf(cc.uz[1], v.y, cc.uz[2]));
            const float dt = softplus20(fmaf(cc.ud[0], v.x, fmaf(cc.ud[1], v.y, cc.ud[2])));
            const float dy = row[36 + j] * silu(z);
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                float abe, abo, cs, sn;
                pair_coeffs(dt, cc.ah[2 * p], cc.ah[2 * p + 1], cc.f[p], abe, abo, cs, sn);
                // M_t^T = [[abe*cs, abo*sn], [-abe*sn, abo*cs]];  P <- P * M_t^T ;  acc += P * (dy*C)
                const float a0 = m[4 * p], b0 = m[4 * p + 1], c0 = m[4 * p + 2], d0 = m[4 * p + 3];
                const float t1 = abe * cs, t2 = abo * sn, t3 = -abe * sn, t4 = abo * cs;
                const float na = fmaf(a0, t1, b0 * t3), nb = fmaf(a0, t2, b0 * t4), nc = fmaf(c0, t1, d0 * t3), nd = fmaf(c0, t2, d0 * t4);
                m[4 * p] = na; m[4 * p + 1] = nb; m[4 * p + 2] = nc; m[4 * p + 3] = nd;
                const float ie = dy * row[16 + row_pos(2 * p)], io = dy * row[16 + row_pos(2 * p + 1)];
                acc[2 * p] = fmaf(na, ie, fmaf(nb, io, acc[2 * p]));
                acc[2 * p + 1] = fmaf(nc, ie, fmaf(nd, io, acc[2 * p + 1]));
            }
        }
        bool zero = true;
#pragma unroll
        for (int k = 0; k < 32; ++k) zero = zero && (fabsf(m[k]) < 7.8886e-31f);
        __syncwarp(hmask);
        if (__all_sync(hmask, zero)) break;
    }
    float* dst = agg + ((int64_t)item_idx * 16 + j) * 48;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        dst[6 * p] = m[4 * p]; dst[6 * p + 1] = m[4 * p + 1]; dst[6 * p + 2] = m[4 * p + 2]; dst[6 * p + 3] = m[4 * p + 3];
        dst[6 * p + 4] = acc[2 * p]; dst[6 * p + 5] = acc[2 * p + 1];
    }
}

__global__ void __launch_bounds__(BL_THREADS) sg2_adj1_kernel(const Item* __restrict__ items, int n_items, int dir1_start,
                                                              const float2* __restrict__ gs, const uint32_t* __restrict__ vals_sorted,
                                                              const float* __restrict__ dctx, float* __restrict__ agg) {
    __shared__ __align__(16) float tiles[BL_ITEMS][BL_TILE * BL_ROW];
    const int slot = threadIdx.x >> 4, j = threadIdx.x & 15;
    const int item_idx = blockIdx.x * BL_ITEMS + slot;
    const unsigned hmask = 0xffffu << (16 * ((threadIdx.x >> 4) & 1));
    if (item_idx >= n_items) return;
    const Item it = items[item_idx];
    if (it.tensor < 0 || it.ub == 0) return;            // the first chunk's aggregate has no consumer
    if (item_idx < dir1_start) bl_adj1<0>(it, gs, vals_sorted, dctx, agg, tiles[slot], item_idx, j, hmask);
    else                       bl_adj1<1>(it, gs, vals_sorted, dctx, agg, tiles[slot], item_idx, j, hmask);
}

// ---- adj 2: dh arriving at the end of every chunk ----
__global__ void __launch_bounds__(128) sg2_adj2_kernel(const TensorDir* __restrict__ tds, const float* __restrict__ agg, float* __restrict__ dcarry) {
    const TensorDir td = tds[blockIdx.x];
    const int j = threadIdx.x >> 3, p = threadIdx.x & 7;
    float de = 0.f, dd = 0.f;                             // nothing flows into the final state
    for (int c = td.nc - 1; c >= 0; --c) {
        const int64_t idx = (int64_t)(td.item0 + c);
        float* co = dcarry + (idx * 16 + j) * 16 + 2 * p;
        co[0] = de; co[1] = dd;
        if (c > 0) {
            const float* a = agg + (idx * 16 + j) * 48 + 6 * p;
            const float ne = fmaf(a[0], de, fmaf(a[1], dd, a[4]));
            const float no = fmaf(a[2], de, fmaf(a[3], dd, a[5]));
            de = ne; dd = no;
        }
    }
}

// Half a column (lane = (half, column j)): four RoPE pairs as two packed groups, see scan_phase3.
struct HalfState { f2 he[2], ho[2]; };
struct HalfConst { f2 ahe[2], aho[2], f[2]; float ux[3], uz[3], ud[3], Dj; };
template <int DIR>
__device__ __forceinline__ void bl_load_const(HalfConst& cc, int j, int half) {
    constexpr int W = (DIR == 0) ? P::DIR0 : P::DIR1;
    constexpr int AF = (DIR == 0) ? P::AFF0 : P::AFF1;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int w = W + P::D_ALOG + j * 16 + 8 * half + 4 * q, r = W + P::D_ROPE + j * 8 + 4 * half + 2 * q;
        cc.ahe[q] = pk(-0.5f * __expf(c_w[w]), -0.5f * __expf(c_w[w + 2]));
        cc.aho[q] = pk(-0.5f * __expf(c_w[w + 1]), -0.5f * __expf(c_w[w + 3]));
        cc.f[q] = pk(c_w[r], c_w[r + 1]);
        asm volatile("" : "+l"(cc.ahe[q]), "+l"(cc.aho[q]), "+l"(cc.f[q]));       // held in registers, see scan_phase3
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        cc.ux[k] = c_w[AF + P::A_X + 3 * j + k]; cc.uz[k] = c_w[AF + P::A_Z + 3 * j + k]; cc.ud[k] = c_w[AF + P::A_DT + 3 * j + k];
        asm volatile("" : "+f"(cc.ux[k]), "+f"(cc.uz[k]), "+f"(cc.ud[k]));
    }
    cc.Dj = c_w[W + P::D_D + j];
    asm volatile("" : "+f"(cc.Dj));
}

// Forward recurrence through the cnt timesteps of one tile (state only), in the arithmetic of the forward scan: a state recomputed from
// a snapshot is bit for bit the one that a snapshot at that place would have held.  HIST: the state BEFORE each step is kept in
// hist[(step * 8 + k) * 32 + lane].
template <bool HIST, int PITCH>
__device__ __forceinline__ void bl_advance(const HalfConst& cc, const float* __restrict__ tile, int cnt, HalfState& h, float* __restrict__ hist, int half, int lane) {
#pragma unroll 1
    for (int l = 0; l < cnt; ++l) {
        const float* row = tile + l * PITCH;
        const float2 v = *reinterpret_cast<const float2*>(row + 32);
        const float x = fmaf(cc.ux[0], v.x, fmaf(cc.ux[1], v.y, cc.ux[2]));
        const float dt = softplus20(fmaf(cc.ud[0], v.x, fmaf(cc.ud[1], v.y, cc.ud[2])));
        const float dtx = dt * x;
        const f2 ndt2 = pk(-dt, -dt), dt2 = pk(dt, dt), dtx2 = pk(dtx, dtx), mone = pk(-1.f, -1.f);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if constexpr (HIST) {
                float e0, e1, o0, o1;
                upk(h.he[q], e0, e1); upk(h.ho[q], o0, o1);
                float* d = hist + (l * 8 + 4 * q) * 32 + lane;
                d[0] = e0; d[32] = o0; d[64] = e1; d[96] = o1;
            }
            const ulonglong2 B = reinterpret_cast<const ulonglong2*>(row + 8 * half)[q];
            f2 abe, abo, cs, sn;
            quad_coeffs(ndt2, dt2, cc.ahe[q], cc.aho[q], cc.f[q], abe, abo, cs, sn);
            const f2 re = fma2(h.ho[q], mul2(sn, mone), mul2(h.he[q], cs)), ro = fma2(h.he[q], sn, mul2(h.ho[q], cs));
            h.he[q] = fma2(abe, re, mul2(dtx2, B.x));
            h.ho[q] = fma2(abo, ro, mul2(dtx2, B.y));
        }
    }
}

// ---- adj 3: the adjoint proper ----
// State snapshots are kept at the start of every `snap_every`-th tile (checkpoint interval = snap_every * BL_TILE timesteps); a tile
// that does not start at a snapshot is reached by re-running the forward recurrence from the snapshot before it, which trades
// (snap_every - 1) / 2 extra tile passes on average for 1 / snap_every of the snapshot memory.  The gradients do not depend on it.
// A warp per chunk: the states before the 16 steps of a tile take 16 KB of shared memory per chunk, which leaves room for ten chunks on
// an SM; with half a warp each that was 1.25 warps per scheduler and latency all the way (422,755 parameters: 1,395 -> 950 us).
template <int DIR>
__device__ void bl_adj3(const Item& it, const float2* __restrict__ gs, const uint32_t* __restrict__ vals_sorted, const float* __restrict__ dctx,
                        const float* __restrict__ dcarry, const float* __restrict__ snaps, int64_t snap_base,
                        float* __restrict__ partial, float* __restrict__ tile, float* __restrict__ hist, int item_idx, int lane, int snap_every) {
    const int j = lane & 15, half = lane >> 4;
    HalfConst cc;
    bl_load_const<DIR>(cc, j, half);
    const int len = it.ue - it.ub;
    const int ntile = (len + BL_TILE - 1) / BL_TILE;
    float ah[8], f[4];                                     // the same constants, one by one (local state k = global state 8 half + k)
#pragma unroll
    for (int q = 0; q < 2; ++q) { upk(cc.ahe[q], ah[4 * q], ah[4 * q + 2]); upk(cc.aho[q], ah[4 * q + 1], ah[4 * q + 3]); upk(cc.f[q], f[2 * q], f[2 * q + 1]); }
    float dh[8], dah[8], df[4], dux[3] = {0.f, 0.f, 0.f}, duz[3] = {0.f, 0.f, 0.f}, dud[3] = {0.f, 0.f, 0.f}, dwo[8], dD = 0.f;
    {
        const float* din = dcarry + ((int64_t)item_idx * 16 + j) * 16 + 8 * half;
#pragma unroll
        for (int q = 0; q < 2; ++q) { const float4 t = reinterpret_cast<const float4*>(din)[q]; dh[4 * q] = t.x; dh[4 * q + 1] = t.y; dh[4 * q + 2] = t.z; dh[4 * q + 3] = t.w; }
    }
#pragma unroll
    for (int s = 0; s < 8; ++s) dah[s] = dwo[s] = 0.f;
#pragma unroll
    for (int p = 0; p < 4; ++p) df[p] = 0.f;
    float dbc[3] = {0.f, 0.f, 0.f};                        // dU_B (j < 8) or dU_C row of state 8 half + (j & 7), summed over the columns
    for (int tI = ntile - 1; tI >= 0; --tI) {
        const int u0 = it.ub + tI * BL_TILE;
        const int cnt = (it.ue - u0 < BL_TILE) ? (it.ue - u0) : BL_TILE;
        HalfState h;
        {   // state at the start of this tile: the snapshot, advanced through the tiles between the snapshot and this one
            const int t0 = tI - tI % snap_every;
            const float* sp = snaps + ((snap_base + t0 / snap_every) * 16 + j) * 16 + 8 * half;
#pragma unroll
            for (int q = 0; q < 2; ++q) { const float4 t = reinterpret_cast<const float4*>(sp)[q]; h.he[q] = pk(t.x, t.z); h.ho[q] = pk(t.y, t.w); }
            for (int t = t0; t < tI; ++t) {                // full tiles (only the last tile of a chunk can be short)
                stage_a<DIR>(tile, gs, it.off, it.n, it.ub + t * BL_TILE + j, half == 0, j);
                __syncwarp();
                bl_advance<false, ROW>(cc, tile, BL_TILE, h, nullptr, half, lane);
                __syncwarp();
            }
        }
        bl_stage_a<DIR>(tile, gs, vals_sorted, dctx, it.off, it.n, u0 + j, half == 0 && j < cnt, j);
        __syncwarp();
        bl_advance<true, BL_ROW>(cc, tile, cnt, h, hist, half, lane);
        // reverse through the tile; the gradients are summed per tile first, so that a chunk of thousands of steps adds a sixteenth as many
        // terms to its large sums
        float tb[3] = {0.f, 0.f, 0.f}, tx[3] = {0.f, 0.f, 0.f}, tz[3] = {0.f, 0.f, 0.f}, td[3] = {0.f, 0.f, 0.f}, tD = 0.f, tah[8], tf[4], two[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) tah[s] = two[s] = 0.f;
#pragma unroll
        for (int p = 0; p < 4; ++p) tf[p] = 0.f;
#pragma unroll 1
        for (int l = cnt - 1; l >= 0; --l) {
            const float* row = tile + l * BL_ROW;
            const float* rb = row + 8 * half;
            const float2 v = *reinterpret_cast<const float2*>(row + 32);
            const float in3[3] = {v.x, v.y, 1.f};
            const float x = fmaf(cc.ux[0], v.x, fmaf(cc.ux[1], v.y, cc.ux[2]));
            const float z = fmaf(cc.uz[0], v.x, fmaf(cc.uz[1], v.y, cc.uz[2]));
            const float dtr = fmaf(cc.ud[0], v.x, fmaf(cc.ud[1], v.y, cc.ud[2]));
            const float dt = softplus20(dtr);
            const float dtx = dt * x;
            const float gout = row[36 + j];
            const float sz = sigmoidf(z), sl = z * sz;
            const float dy = gout * sl;
            float y = 0.f, ddt = 0.f, ddtx = 0.f, v16[16];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int e = 2 * p, o = 2 * p + 1;
                float abe, abo, cs, sn;
                pair_coeffs(dt, ah[e], ah[o], f[p], abe, abo, cs, sn);
                const float he = hist[(l * 8 + e) * 32 + lane], ho = hist[(l * 8 + o) * 32 + lane];
                const float re = he * cs - ho * sn, ro = ho * cs + he * sn;
                const float Be = rb[row_pos(e)], Bo = rb[row_pos(o)], Ce = rb[16 + row_pos(e)], Co = rb[16 + row_pos(o)];
                const float hce = fmaf(abe, re, dtx * Be), hco = fmaf(abo, ro, dtx * Bo);     // state AFTER this step
                y = fmaf(hce, Ce, fmaf(hco, Co, y));
                const float de = fmaf(dy, Ce, dh[e]), dd = fmaf(dy, Co, dh[o]);
                v16[e] = de * dtx; v16[o] = dd * dtx; v16[8 + e] = dy * hce; v16[8 + o] = dy * hco;      // d B, d C of this column
                ddtx = fmaf(de, Be, fmaf(dd, Bo, ddtx));
                const float dabe = de * re, dabo = dd * ro, dre = de * abe, dro = dd * abo;
                const float dcs = fmaf(dre, he, dro * ho), dsn = fmaf(dro, he, -dre * ho);
                const float dth = fmaf(cs, dsn, -sn * dcs);
                ddt = fmaf(dth, f[p], ddt);
                tf[p] = fmaf(dth, dt, tf[p]);
                const float gae = dabe * (abe + 1.f) * (abe + 1.f) * 0.5f, gao = dabo * (abo + 1.f) * (abo + 1.f) * 0.5f;
                ddt = fmaf(gae, ah[e], fmaf(gao, ah[o], ddt));
                tah[e] = fmaf(gae, dt, tah[e]); tah[o] = fmaf(gao, dt, tah[o]);
                dh[e] = fmaf(dre, cs, dro * sn);
                dh[o] = fmaf(dro, cs, -dre * sn);
            }
            y += __shfl_xor_sync(0xffffffffu, y, 16);         // both halves of the column
            ddt += __shfl_xor_sync(0xffffffffu, ddt, 16);
            ddtx += __shfl_xor_sync(0xffffffffu, ddtx, 16);
            {   // d B and d C are shared by the sixteen columns: halve the 16 values four times over the lanes, lane j ends with one sum
                float r8[8], r4[4], r2[2];
                const bool b3 = j & 8, b2 = j & 4, b1 = j & 2, b0 = j & 1;
#pragma unroll
                for (int k = 0; k < 8; ++k) r8[k] = (b3 ? v16[8 + k] : v16[k]) + __shfl_xor_sync(0xffffffffu, b3 ? v16[k] : v16[8 + k], 8);
#pragma unroll
                for (int k = 0; k < 4; ++k) r4[k] = (b2 ? r8[4 + k] : r8[k]) + __shfl_xor_sync(0xffffffffu, b2 ? r8[k] : r8[4 + k], 4);
#pragma unroll
                for (int k = 0; k < 2; ++k) r2[k] = (b1 ? r4[2 + k] : r4[k]) + __shfl_xor_sync(0xffffffffu, b1 ? r4[k] : r4[2 + k], 2);
                const float t = (b0 ? r2[1] : r2[0]) + __shfl_xor_sync(0xffffffffu, b0 ? r2[0] : r2[1], 1);
                tb[0] = fmaf(t, in3[0], tb[0]); tb[1] = fmaf(t, in3[1], tb[1]); tb[2] += t;
            }
            const float outj = fmaf(y, sl, cc.Dj * x);
            const float dz = gout * y * sz * (1.f + z * (1.f - sz));
            tD = fmaf(gout, x, tD);
            const float dx = fmaf(gout, cc.Dj, ddtx * dt);
            ddt = fmaf(ddtx, x, ddt);
            const float ddtr = ddt * (dtr > 20.f ? 1.f : sigmoidf(dtr));
#pragma unroll
            for (int k = 0; k < 3; ++k) { tx[k] = fmaf(dx, in3[k], tx[k]); tz[k] = fmaf(dz, in3[k], tz[k]); td[k] = fmaf(ddtr, in3[k], td[k]); }
#pragma unroll
            for (int d = 0; d < 8; ++d) two[d] = fmaf(row[52 + d], outj, two[d]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) { dbc[k] += tb[k]; dux[k] += tx[k]; duz[k] += tz[k]; dud[k] += td[k]; }
#pragma unroll
        for (int s = 0; s < 8; ++s) { dah[s] += tah[s]; dwo[s] += two[s]; }
#pragma unroll
        for (int p = 0; p < 4; ++p) df[p] += tf[p];
        dD += tD;
        __syncwarp();
    }
    // ---- per-item partial gradients: [item][BL_NG]
    float* out = partial + (int64_t)item_idx * BL_NG;
#pragma unroll
    for (int s = 0; s < 8; ++s) out[j * 16 + 8 * half + s] = dah[s];    // d(A/2); converted to d A_log by the reduction kernel
#pragma unroll
    for (int p = 0; p < 4; ++p) out[256 + j * 8 + 4 * half + p] = df[p];
#pragma unroll
    for (int c = 0; c < 3; ++c) out[544 + ((j >> 3) * 16 + 8 * half + (j & 7)) * 3 + c] = dbc[c];
    if (half == 0) {                                                     // both halves hold the column's own sums
        out[384 + j] = dD;
#pragma unroll
        for (int k = 0; k < 3; ++k) { out[400 + j * 3 + k] = dux[k]; out[448 + j * 3 + k] = duz[k]; out[496 + j * 3 + k] = dud[k]; }
#pragma unroll
        for (int d = 0; d < 8; ++d) out[640 + d * 16 + j] = dwo[d];
    }
}

__global__ void __launch_bounds__(32) sg2_adj3_kernel(const Item* __restrict__ items, int n_items, int dir1_start,
                                                      const int64_t* __restrict__ snap_base, const float2* __restrict__ gs,
                                                      const uint32_t* __restrict__ vals_sorted, const float* __restrict__ dctx,
                                                      const float* __restrict__ dcarry, const float* __restrict__ snaps,
                                                      float* __restrict__ partial, int snap_every) {
    __shared__ __align__(16) float tile[BL_TILE * BL_ROW];              // BL_ROW >= ROW
    __shared__ float hist[BL_TILE * 8 * 32];
    const int item_idx = blockIdx.x, lane = threadIdx.x;
    const Item it = items[item_idx];
    if (it.tensor < 0) {
        for (int k = lane; k < BL_NG; k += 32) partial[(int64_t)item_idx * BL_NG + k] = 0.f;
        return;
    }
    if (item_idx < dir1_start) bl_adj3<0>(it, gs, vals_sorted, dctx, dcarry, snaps, snap_base[item_idx], partial, tile, hist, item_idx, lane, snap_every);
    else                       bl_adj3<1>(it, gs, vals_sorted, dctx, dcarry, snaps, snap_base[item_idx], partial, tile, hist, item_idx, lane, snap_every);
}

// ---- adj 4: fixed-order sum over the items of each direction; d(A/2) -> d A_log ----
__global__ void __launch_bounds__(1024) sg2_adj4_kernel(const float* __restrict__ partial, int n_items, int dir1_start, float* __restrict__ grads) {
    const int dir = blockIdx.y, k = blockIdx.x * 32 + (threadIdx.x & 31);
    float s = column_parts_sum(partial, dir == 0 ? 0 : dir1_start, dir == 0 ? dir1_start : n_items, BL_NG, k);
    if (threadIdx.x >= 32 || k >= BL_NG) return;
    if (k < 256) {                                                      // ah = -0.5*exp(A_log)  =>  d A_log = d ah * ah
        const int W = (dir == 0) ? P::DIR0 : P::DIR1;
        s *= -0.5f * __expf(c_w[W + P::D_ALOG + k]);
    }
    grads[dir * BL_NG + k] = s;
}

}  // namespace

int sg2_bilevel_ng() { return BL_NG; }
int sg2_bilevel_tile() { return BL_TILE; }

// dctx [total,16] (original order) -> grads [2][BL_NG].  Uses agg / dcarry scratch of the sizes of the forward's agg / carry, the states that
// the forward scan has left in snaps [sum over items of ceil(tiles / snap_every), 16, 16] and
// partial [n_items, BL_NG].  snap_base[item] = index of the item's first snapshot.
void sg2_scan_backward(const void* items_dev, int n_items, int dir1_start, const void* tds_dev, int n_td, const int64_t* snap_base_dev,
                       const float* gs_sorted, const uint32_t* vals_sorted, const float* dctx, float* agg, float* dcarry,
                       float* snaps, float* partial, float* grads, int snap_every, cudaStream_t s) {
    if (n_items <= 0) return;
    if (snap_every < 1) snap_every = 1;
    const Item* items = reinterpret_cast<const Item*>(items_dev);
    const TensorDir* tds = reinterpret_cast<const TensorDir*>(tds_dev);
    const float2* gs = reinterpret_cast<const float2*>(gs_sorted);
    const int blocks = (n_items + BL_ITEMS - 1) / BL_ITEMS;
    count_launch(4);
    sg2_adj1_kernel<<<blocks, BL_THREADS, 0, s>>>(items, n_items, dir1_start, gs, vals_sorted, dctx, agg);
    sg2_adj2_kernel<<<n_td, 128, 0, s>>>(tds, agg, dcarry);
    sg2_adj3_kernel<<<n_items, 32, 0, s>>>(items, n_items, dir1_start, snap_base_dev, gs, vals_sorted, dctx, dcarry, snaps, partial, snap_every);
    sg2_adj4_kernel<<<dim3((BL_NG + 31) / 32, 2), 1024, 0, s>>>(partial, n_items, dir1_start, grads);
}

}  // namespace sg
