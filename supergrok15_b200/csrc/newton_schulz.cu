// Newton-Schulz iteration of Muon for ALL matrices of a step at once (sm_100a).
//
//   X <- aX + b(XX^T)X + c(XX^T)^2 X     per matrix, `steps` times, as three products on the short side n = min(r, c):
//   G = X X^T (r < c) or X^T X;   P = aI + bG + cG^2;   X <- P X or X P
//
// Each product is ONE persistent launch over the tiles of every matrix: a parameter list has a handful of distinct shapes, the
// matrices of a shape lie one after the other in the workspace and share 3-D tensor maps, and the maps of all shapes travel as kernel
// parameters (no descriptor upload, nothing that outlives the launch).  One launch per matrix and product kept 2 to 16 of the
// 148 SMs busy for ~26 us at d = 256: 240 launches, 6.4 ms for the sixteen matrices of the 4-layer d256 decoder.
//
// What each product saves over a plain GEMM:
//   * X is read where it is in both roles (K-major or MN-major shared-memory descriptors, chosen per shape), so no X^T exists;
//   * G and P are symmetric: only the tiles on and above the block diagonal are computed, the others are written as the transposed
//     copy of their mirror tile (a second, transposed TMA store from shared memory).
// Measured, whole Muon step before -> now: sixteen matrices of the d256 decoder 6.1 ms -> 0.18 ms (bound by fifteen dependent short
// launches of ~9 us), fourteen matrices of two d2048 / 5504 blocks 10.2 ms -> 4.4 ms (the products 3.2 ms at 1.1 PFLOP/s issued,
// 3.7 TFLOP instead of 5.3; bound by the tensor pipe under the power cap).
// Roles, ring and TMEM double buffering are those of gemm_sm100.cu: warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 epilogue.
#include <cuda_fp16.h>
#include "sg_native.h"
#include "newton_schulz.h"
#include "per_device.h"
#include "optim_math.cuh"
#include "tc_sm100.cuh"

namespace sg {
namespace {
using namespace tc;

constexpr int BM = 128, BK = 64;
constexpr int NS_THREADS = 192;
// Shapes per launch.  A launch copies its whole parameter block (576 bytes per shape), and the short products of small models are
// bound by how fast launches follow one another, so parameter lists with few shapes (a decoder has four) take the small block.
constexpr int NS_GROUPS = 40, NS_FEW = 6;

struct alignas(64) NsProblem {
    CUtensorMap a, b, c, ct;                      // operands, output, output seen transposed (symmetric products)
    const __nv_bfloat16* d;                       // C = alpha * acc + beta * D + diag * I (same layout as C), or null
    int ldd;
    int M, N, K, batch;
    int tile0, tiles;                             // first tile in the launch, tiles of one matrix
    int a_mn, b_mn, sym, c_f32;
};
static_assert(sizeof(NsProblem) == 576, "four tensor maps of 128 bytes and the sizes");
template <int CAP> struct NsArgs {
    NsProblem p[CAP];
    int n, total;
    float alpha, beta, diag;
};

// Tiles of a symmetric [n, n] product: square blocks of max(BM, BN) on and above the diagonal, cut into BM x BN tiles.
__host__ __device__ inline int ns_sym_tiles(int n, int bn) {
    const int S = bn > BM ? bn : BM, nb = (n + S - 1) / S;
    return nb * (nb + 1) / 2 * (S / BM) * (S / bn);
}
// (m0, n0) of tile t; `mirror`: the tile lies above the block diagonal and its transpose has to be written as well
__host__ __device__ inline void ns_sym_coords(int t, int bn, int& m0, int& n0, bool& mirror) {
    const int S = bn > BM ? bn : BM, sub = (S / BM) * (S / bn);
    const int blk = t / sub, k = t % sub;
    int bj = (int)((sqrtf(8.f * blk + 1.f) - 1.f) * 0.5f);
    while (bj * (bj + 1) / 2 > blk) --bj;
    while ((bj + 1) * (bj + 2) / 2 <= blk) ++bj;
    const int bi = blk - bj * (bj + 1) / 2;
    m0 = bi * S + (S > BM ? k * BM : 0);
    n0 = bj * S + (S > bn ? k * bn : 0);
    mirror = bi != bj;
}
// Tiles of a general product: groups of 16 tile rows, m fastest (the order of gemm_sm100.cu, so that tiles in flight share panels).
__host__ __device__ inline void ns_plain_coords(int t, int tiles_m, int tiles_n, int bn, int& m0, int& n0) {
    const int per = 16 * tiles_n, first = (t / per) * 16, gsz = tiles_m - first < 16 ? tiles_m - first : 16, r = t % per;
    m0 = (first + r % gsz) * BM;
    n0 = (r / gsz) * bn;
}

struct NsTile { const NsProblem* p; int z, m0, n0; bool mirror; };
template <int BN, typename Args>
__device__ __forceinline__ NsTile ns_tile(const Args& g, int tile) {
    int k = 0;
    while (k + 1 < g.n && g.p[k + 1].tile0 <= tile) ++k;
    NsTile t;
    t.p = &g.p[k];
    const int rel = tile - t.p->tile0, in = rel % t.p->tiles;
    t.z = rel / t.p->tiles;
    t.mirror = false;
    if (t.p->sym) ns_sym_coords(in, BN, t.m0, t.n0, t.mirror);
    else ns_plain_coords(in, (t.p->M + BM - 1) / BM, (t.p->N + BN - 1) / BN, BN, t.m0, t.n0);
    return t;
}

template <int BN, int STAGES, int CAP>
__global__ void __launch_bounds__(NS_THREADS, 1) ns_gemm_kernel(const __grid_constant__ NsArgs<CAP> g, int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr uint32_t A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr uint32_t STG = 32 * 128;                               // staging buffer: 32 rows x 128 bytes (or 64 x 64 transposed)
    uint8_t* staging = smem + STAGES * STAGE_BYTES;                   // [4 warps][2][STG]
    uint64_t* full = reinterpret_cast<uint64_t*>(staging + 4 * 2 * STG);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;                              // [2]
    uint64_t* acc_empty = acc_full + 2;                               // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)(2 * BN)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Launched programmatically: the next product's CTAs may be set up as soon as these leave their SMs, and none of them touches
    // global memory before this wait has seen the whole previous product.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < g.total; tile += gridDim.x) {
                const NsTile t = ns_tile<BN>(g, tile);
                const NsProblem& p = *t.p;
                if (t.m0 >= p.M || t.n0 >= p.N) continue;             // every role skips the same tiles
                const int KB = (p.K + BK - 1) / BK;                   // past the end of K the boxes are zero-filled
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (it >= (uint32_t)STAGES && !mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1)) { atomicExch(err, 21); ok = false; break; }
                    uint8_t* dst = smem + s * STAGE_BYTES;
                    mbar_expect_tx(&full[s], STAGE_BYTES);
                    if (p.a_mn) {
#pragma unroll
                        for (int c = 0; c < BM / 64; ++c) tma_load_3d(dst + c * (BK * 128), &p.a, t.m0 + 64 * c, kb * BK, t.z, &full[s]);
                    } else tma_load_3d(dst, &p.a, kb * BK, t.m0, t.z, &full[s]);
                    if (p.b_mn) {
#pragma unroll
                        for (int c = 0; c < BN / 64; ++c) tma_load_3d(dst + A_BYTES + c * (BK * 128), &p.b, t.n0 + 64 * c, kb * BK, t.z, &full[s]);
                    } else tma_load_3d(dst + A_BYTES, &p.b, kb * BK, t.n0, t.z, &full[s]);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t it = 0, n_acc = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < g.total; tile += gridDim.x) {
                const NsTile t = ns_tile<BN>(g, tile);
                const NsProblem& p = *t.p;
                if (t.m0 >= p.M || t.n0 >= p.N) continue;
                const uint32_t buf = n_acc & 1;
                if (n_acc >= 2 && !mbar_wait(&acc_empty[buf], ((n_acc >> 1) & 1) ^ 1)) { atomicExch(err, 24); ok = false; }
                ++n_acc;
                tc_fence_after();
                const bool a_mn = p.a_mn != 0, b_mn = p.b_mn != 0;
                const uint32_t idesc = make_idesc_bf16(BM, BN, a_mn ? 1 : 0, b_mn ? 1 : 0);
                // descriptor step per 16-wide K slice: 32 bytes along a K-major row, 16 rows of 128 bytes of an MN-major chunk
                const uint64_t sa = a_mn ? 128 : 2, sb = b_mn ? 128 : 2;
                const uint32_t tmem_d = tmem_base + buf * BN;
                const int KB = (p.K + BK - 1) / BK;
                for (int kb = 0; kb < KB && ok; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(&full[s], (it / STAGES) & 1)) { atomicExch(err, 22); ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * STAGE_BYTES);
                    const uint64_t da = a_mn ? make_desc_sw128_mn(a_addr, BK * 128, 1024) : make_desc_sw128(a_addr);
                    const uint64_t db = b_mn ? make_desc_sw128_mn(a_addr + A_BYTES, BK * 128, 1024) : make_desc_sw128(a_addr + A_BYTES);
#pragma unroll
                    for (int k4 = 0; k4 < BK / 16; ++k4) tc_mma_bf16(tmem_d, da + sa * k4, db + sb * k4, idesc, (kb > 0 || k4 > 0) ? 1u : 0u);
                    tc_commit(&empty[s]);
                }
                tc_commit(&acc_full[buf]);                            // also arrives when bailing out
            }
        }
    } else {
        const int q = warp & 3;                                       // TMEM lane quarter of this warp
        uint8_t* stg = staging + (warp - 2) * 2 * STG;
        uint32_t n_acc = 0, sbuf = 0;
        for (int tile = blockIdx.x; tile < g.total; tile += gridDim.x) {
            const NsTile t = ns_tile<BN>(g, tile);
            const NsProblem& p = *t.p;
            if (t.m0 >= p.M || t.n0 >= p.N) continue;
            const uint32_t buf = n_acc & 1;
            const uint32_t parity = (n_acc >> 1) & 1;
            ++n_acc;
            const int row = t.m0 + q * 32 + lane;
            const __nv_bfloat16* drow = p.d != nullptr && row < p.M ? p.d + ((int64_t)t.z * p.M + row) * p.ldd : nullptr;
            if (!mbar_wait(&acc_full[buf], parity)) { if (lane == 0) atomicExch(err, 23); break; }
            tc_fence_after();
            const bool plain = p.d == nullptr;
            const int cols_per_box = p.c_f32 ? 32 : 64;               // 128 bytes of output per row
#pragma unroll 1
            for (int c = 0; c < BN; c += cols_per_box) {
                if (t.n0 + c >= p.N) break;
                // The buffer about to be written must have been read by its TMA store: with two buffers in turn that is all but the
                // newest store; a symmetric product uses the second buffer for the transposed copy, so all of them.
                if (lane == 0) {
                    if (p.sym) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                }
                __syncwarp();
                uint8_t* sb = stg + (p.sym ? 0 : sbuf * STG);
                uint8_t* st = stg + STG;                              // transposed copy: 64 rows (output columns) x 32 rows of C, dense
#pragma unroll 1
                for (int h = 0; h < cols_per_box; h += 32) {
                    const int col0 = t.n0 + c + h;
                    uint4 dv[4];
                    if (drow) {                                       // rows are padded to 8 elements: a group that starts inside N is readable
#pragma unroll
                        for (int k = 0; k < 4; ++k) if (col0 + 8 * k < p.N) dv[k] = *reinterpret_cast<const uint4*>(drow + col0 + 8 * k);
                    }
                    uint32_t r[32];
                    tc_ld32(tmem_base + buf * BN + ((uint32_t)(q * 32) << 16) + (uint32_t)(c + h), r);
                    tc_wait_ld();
                    if (!plain) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const __nv_bfloat162* dh = reinterpret_cast<const __nv_bfloat162*>(&dv[k]);
                            const bool have = drow != nullptr && col0 + 8 * k < p.N;
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const float2 f = have ? __bfloat1622float2(dh[u]) : make_float2(0.f, 0.f);
                                r[8 * k + 2 * u] = __float_as_uint(fmaf(g.beta, f.x, g.alpha * __uint_as_float(r[8 * k + 2 * u])));
                                r[8 * k + 2 * u + 1] = __float_as_uint(fmaf(g.beta, f.y, g.alpha * __uint_as_float(r[8 * k + 2 * u + 1])));
                            }
                        }
                        const int dj = row - col0;                    // the identity of this lane's row, if it lies in these 32 columns
#pragma unroll
                        for (int j = 0; j < 32; ++j) if (j == dj) r[j] = __float_as_uint(__uint_as_float(r[j]) + g.diag);
                    }
                    // 16-byte chunk k of row `lane` lives at chunk k ^ (lane & 7) of the swizzled staging row
                    uint8_t* rowp = sb + lane * 128;
                    if (p.c_f32) {
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            *reinterpret_cast<uint4*>(rowp + ((k ^ (lane & 7)) << 4)) = make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            uint4 o;
                            __nv_bfloat162* hh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                            for (int u = 0; u < 4; ++u) hh[u] = __floats2bfloat162_rn(__uint_as_float(r[8 * k + 2 * u]), __uint_as_float(r[8 * k + 2 * u + 1]));
                            *reinterpret_cast<uint4*>(rowp + ((((h >> 3) + k) ^ (lane & 7)) << 4)) = o;
                            if (t.mirror) {                           // lanes write 64 consecutive bytes per column: no bank conflict
#pragma unroll
                                for (int u = 0; u < 4; ++u) {
                                    *reinterpret_cast<__nv_bfloat16*>(st + (h + 8 * k + 2 * u) * 64 + lane * 2) = hh[u].x;
                                    *reinterpret_cast<__nv_bfloat16*>(st + (h + 8 * k + 2 * u + 1) * 64 + lane * 2) = hh[u].y;
                                }
                            }
                        }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    tma_store_3d(&p.c, sb, t.n0 + c, t.m0 + q * 32, t.z);
                    if (t.mirror) tma_store_3d(&p.ct, st, t.m0 + q * 32, t.n0 + c, t.z);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                sbuf ^= 1;
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * BN)) : "memory");
    }
}

// X = buf * inv, rounded to bf16, into the padded workspace rows.  One pass over all matrices (it replaced a multiply, two casts, a
// transpose and four fills per matrix); a CTA takes NS_CAST elements of one matrix.
constexpr int NS_CAST = 8192;
struct NsCastArgs {
    const float* src[MT_MAX];
    __nv_bfloat16* dst[MT_MAX];
    int64_t numel[MT_MAX];
    int cols[MT_MAX], ld[MT_MAX];
    int blk0[MT_MAX + 1];
    const float* inv;                             // per-matrix scale, or null (1)
    int n, t_off;
};
__global__ void __launch_bounds__(256) ns_cast_kernel(const __grid_constant__ NsCastArgs a) {
    int lo = 0, hi = a.n;
    while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (a.blk0[mid] <= (int)blockIdx.x) lo = mid; else hi = mid; }
    const int t = lo;
    const float inv = a.inv ? a.inv[a.t_off + t] : 1.f;
    const float* src = a.src[t];
    __nv_bfloat16* dst = a.dst[t];
    const int cols = a.cols[t], ld = a.ld[t];
    const int64_t begin = (int64_t)(blockIdx.x - a.blk0[t]) * NS_CAST, n = a.numel[t];
    const int64_t end = begin + NS_CAST < n ? begin + NS_CAST : n;
    if (cols == ld && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {         // rows without padding: the matrix is one dense run of 8-element groups
        for (int64_t i = begin + threadIdx.x * 8; i < end; i += 256 * 8) {
            const float4 u = *reinterpret_cast<const float4*>(src + i), v = *reinterpret_cast<const float4*>(src + i + 4);
            uint4 o;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
            h[0] = __floats2bfloat162_rn(u.x * inv, u.y * inv); h[1] = __floats2bfloat162_rn(u.z * inv, u.w * inv);
            h[2] = __floats2bfloat162_rn(v.x * inv, v.y * inv); h[3] = __floats2bfloat162_rn(v.z * inv, v.w * inv);
            *reinterpret_cast<uint4*>(dst + i) = o;
        }
    } else {
        for (int64_t i = begin + threadIdx.x; i < end; i += 256) {
            const int64_t row = i / cols;
            dst[row * ld + (i - row * cols)] = __float2bfloat16_rn(src[i] * inv);
        }
    }
}

// One product over all groups.  phase 0: G, 1: P, 2: X (into xn, or out32 when `last`)
struct NsView { const void* base; int64_t rows, cols, ld; bool mn; };

int ns_tiles_of(int M, int N, bool sym, int bn) { return sym ? ns_sym_tiles(M, bn) : ((M + BM - 1) / BM) * ((N + bn - 1) / bn); }

template <int BN, int STAGES, int CAP>
int ns_go(const NsArgs<CAP>& g, int* err, cudaStream_t s) {
    constexpr size_t smem = (size_t)STAGES * (BM * BK * 2 + BN * BK * 2) + 4 * 2 * 4096 + 1024 + 256;
    static std::atomic<uint64_t> granted{0};
    if (!once_per_device(granted, current_device(), [&] {
            return cudaFuncSetAttribute(ns_gemm_kernel<BN, STAGES, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
        })) return 2;
    const int sms = device_sms();
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(g.total < sms ? g.total : sms));
    cfg.blockDim = dim3(NS_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, ns_gemm_kernel<BN, STAGES, CAP>, g, err) == cudaSuccess ? 0 : 3;
}

// Width of the output tiles: the widest that still gives every SM a tile.  256 columns read the least shared memory per MMA;
// where the products are too few or too small to fill the GPU, narrower tiles spread the same work over more SMs.
int ns_pick_bn(const NsGroup* gr, int n, int phase) {
    const int sms = device_sms();
    for (int bn = 256; bn > 64; bn /= 2) {
        int64_t tiles = 0;
        for (int i = 0; i < n; ++i) {
            const int k = gr[i].r < gr[i].c ? gr[i].r : gr[i].c;
            tiles += (int64_t)gr[i].batch * (phase < 2 ? ns_tiles_of(k, k, true, bn) : ns_tiles_of(gr[i].r, gr[i].c, false, bn));
        }
        if (tiles >= sms) return bn;
    }
    return 64;
}

template <int CAP>
int ns_product(const NsGroup* gr, int n, int phase, bool last, int cur, float a, float b, float c, int* err, cudaStream_t s) {
    const int bn = ns_pick_bn(gr, n, phase);
    NsArgs<CAP> g{};
    g.n = n;
    g.alpha = phase == 1 ? c : 1.f;
    g.beta = phase == 1 ? b : 0.f;
    g.diag = phase == 1 ? a : 0.f;
    int64_t total = 0;
    for (int i = 0; i < n; ++i) {
        const NsGroup& q = gr[i];
        NsProblem& p = g.p[i];
        const bool tall = q.r >= q.c;
        const int k = tall ? q.c : q.r, ldk = (k + 7) / 8 * 8, ldx = (q.c + 7) / 8 * 8;
        const void* x = cur ? q.x1 : q.x0;
        void* xn = cur ? q.x0 : q.x1;
        NsView A{x, q.r, q.c, ldx, false}, B = A;
        void* out = q.g;
        p.sym = phase < 2;
        p.batch = q.batch;
        if (phase == 0) {                         // tall: X^T X, both operands read along their rows (MN-major)
            p.M = p.N = k; p.K = tall ? q.r : q.c;
            A.mn = B.mn = tall;
        } else if (phase == 1) {
            A = B = NsView{q.g, k, k, ldk, false};
            p.M = p.N = p.K = k;
            p.d = q.g; p.ldd = ldk;
            out = q.p;
        } else {
            const NsView Pm{q.p, k, k, ldk, false};
            p.M = q.r; p.N = q.c; p.K = k;
            if (tall) B = Pm;                     // X P: P is symmetric, its rows are the columns that B wants
            else { A = Pm; B.mn = true; }         // P X: X is [K, N]
            out = last ? static_cast<void*>(q.out32) : xn;
            p.c_f32 = last;
        }
        p.a_mn = A.mn; p.b_mn = B.mn;
        const int ldo = phase < 2 ? ldk : last ? (q.c + 3) / 4 * 4 : ldx;
        if (!make_map_batched(&p.a, A.base, q.batch, A.rows, A.cols, A.ld, A.mn ? BK : BM, 64, true, true)) return 1;
        if (!make_map_batched(&p.b, B.base, q.batch, B.rows, B.cols, B.ld, B.mn ? BK : bn, 64, true, true)) return 1;
        if (!make_map_batched(&p.c, out, q.batch, p.M, p.N, ldo, 32, p.c_f32 ? 32 : 64, !p.c_f32, true)) return 4;
        if (p.sym && !make_map_batched(&p.ct, out, q.batch, p.N, p.M, ldo, 64, 32, true, false)) return 4;
        p.tile0 = (int)total;
        p.tiles = ns_tiles_of(p.M, p.N, p.sym, bn);
        total += (int64_t)p.tiles * q.batch;
        if (total > 0x7fffffff) return 6;
    }
    g.total = (int)total;
    if (bn == 256) return ns_go<256, 4, CAP>(g, err, s);
    if (bn == 128) return ns_go<128, 6, CAP>(g, err, s);
    return ns_go<64, 8, CAP>(g, err, s);
}

}  // namespace

void ns_sym_tile_coords(int tile, int bn, int* m0, int* n0, int* mirror) {
    bool m;
    ns_sym_coords(tile, bn, *m0, *n0, m);
    *mirror = m;
}
int ns_sym_tile_count(int n, int bn) { return ns_sym_tiles(n, bn); }

void ns_cast(const float* const* src, void* const* dst, const int* rows, const int* cols, int n, const float* inv, cudaStream_t s) {
    for (int t0 = 0; t0 < n; t0 += MT_MAX) {
        NsCastArgs a{};
        a.n = n - t0 < MT_MAX ? n - t0 : MT_MAX;
        a.t_off = t0; a.inv = inv;
        for (int t = 0; t < a.n; ++t) {
            a.src[t] = src[t0 + t];
            a.dst[t] = reinterpret_cast<__nv_bfloat16*>(dst[t0 + t]);
            a.cols[t] = cols[t0 + t]; a.ld[t] = (cols[t0 + t] + 7) / 8 * 8;
            a.numel[t] = (int64_t)rows[t0 + t] * cols[t0 + t];
            a.blk0[t + 1] = a.blk0[t] + (int)((a.numel[t] + NS_CAST - 1) / NS_CAST);
        }
        if (a.blk0[a.n] == 0) continue;
        count_launch();
        ns_cast_kernel<<<a.blk0[a.n], 256, 0, s>>>(a);
    }
}

int ns_iterate(const NsGroup* groups, int n, int steps, float a, float b, float c, int* err, cudaStream_t s) {
    for (int g0 = 0; g0 < n; g0 += NS_GROUPS) {
        const int m = n - g0 < NS_GROUPS ? n - g0 : NS_GROUPS;
        for (int it = 0, cur = 0; it < steps; ++it, cur ^= 1)
            for (int phase = 0; phase < 3; ++phase) {
                const int rc = m <= NS_FEW ? ns_product<NS_FEW>(groups + g0, m, phase, it == steps - 1, cur, a, b, c, err, s)
                                           : ns_product<NS_GROUPS>(groups + g0, m, phase, it == steps - 1, cur, a, b, c, err, s);
                if (rc) return rc;
            }
    }
    return 0;
}

}  // namespace sg
