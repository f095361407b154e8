// The confidence-weighted, edge-aware WLS depth solve (crates/lapstack-core/
// src/depth.rs:958 `WlsSolver`) on the device: the separable fast-global-
// smoother guess (depth.rs:677/707 Thomas sweeps, depth.rs:1022-1034
// schedule), then CG on (W + lambda L) u = W d preconditioned by one V-cycle
// of the 2x2-aggregation multigrid hierarchy (depth.rs:753-947), stopping at
// a relative residual of 1e-5. The f32 stencil, smoother, restriction and
// prolongation follow the reference's operation order; the CG dot products
// are f64 sums in a fixed two-stage order.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <functional>
#include <type_traits>
#include <vector>

#include "lsb_common.cuh"
#include "lsb_depth.h"

namespace lsb {
namespace cg = cooperative_groups;

constexpr float MG_OMEGA = 0.8f;
constexpr int MG_COARSE = 32, MG_MIN = 16;
// the BF16 V-cycle: levels, and Jacobi sweeps before and after the coarse correction
constexpr int MG_H_LEVELS = 6, MG_H_SWEEPS = 2;
// blocks of the element-wise kernels that reduce: 8 of 256 threads an SM
constexpr int RED_BLOCKS = 148 * 8;

struct WlsSolver {
    int w, h;
    float lambda;
    float *ex, *ey;
    std::vector<WlsLevel> lv;
    float *cp, *dp, *f, *r, *z, *p, *p2, *ap;  // p, p2: the search direction, in turn (f: the start sweeps' row results)
    double *part, *scal;  // partial sums of the reductions; scal: [rz, |b|]
    float* alpha_beta;    // [alpha, beta]
    int* ctl;             // [stop, iterations done, blocks of a reduction that are done, p.Ap <= 0]
    bool ctl_zero = false;
    float* host_rel;      // page-locked: [rel, stop, iterations, -, rel as a double]
    const float* guide = nullptr;  // of the last wls_prepare, its edge weights made by the next wls_set_weights
    float inv = 0.f, inv2s2 = 0.f;
    int edge_mode = 0;
    void* slab = nullptr;  // every plane: one allocation
    size_t bytes = 0;
    // one CG iteration as a graph, captured on the first solve for this u and V-cycle mode
    cudaGraphExec_t g = nullptr;
    const float* g_u = nullptr;
    int g_mode = -1, g_max = 0;
    long long g_kernels = 0;
    cudaEvent_t done[2] = {nullptr, nullptr};  // the last two iterations queued
};

static int g1(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 148 * 16); }
static dim3 g2(int w, int h) { return dim3((w + 31) / 32, (h + 7) / 8); }
static const dim3 B2(32, 8);

// BF16 copies of a level's operators (wd, ax, ay, dinv), for the mixed-precision V-cycle; null: none.
struct HOps {
    uint16_t *wd, *ax, *ay, *dinv;
};
typedef __nv_bfloat16 bf;
__device__ __forceinline__ float ldh(const uint16_t* p, size_t k) { return __bfloat162float(((const bf*)p)[k]); }
__device__ __forceinline__ void sth(uint16_t* p, size_t k, float v) { ((bf*)p)[k] = __float2bfloat16_rn(v); }
__device__ __forceinline__ void put_ops(const HOps& H, size_t k, float wd, float ax, float ay, float dinv) {
    if (!H.wd) return;
    sth(H.wd, k, wd);
    sth(H.ax, k, ax);
    sth(H.ay, k, ay);
    sth(H.dinv, k, dinv);
}
// depth.rs:812 `set_dinv` of one cell: its weight and the edges that leave it (0 past the border: adding it changes nothing)
__device__ __forceinline__ float dinv_of(float wd, bool l, float axl, bool r, float axr, bool t, float ayt, bool b, float ayb) {
    float v = wd;
    if (l) v = __fadd_rn(v, axl);
    if (r) v = __fadd_rn(v, axr);
    if (t) v = __fadd_rn(v, ayt);
    if (b) v = __fadd_rn(v, ayb);
    return __fdiv_rn(1.f, fmaxf(v, 1e-12f));
}
// Level 0 of a solve in one pass: depth.rs:653 `edge_weights`, e = exp(-|dI| / sigma) right and below (mode 0; mode 1:
// the Gaussian-of-gradient weight exp(-dI^2 / (2 sigma^2))) times lambda, depth.rs:994 wd = max(conf, 0) + 1e-4 and
// depth.rs:812 the diagonal, the left and upper edges computed again by the cell that needs them. EDGES false: other
// weights on the same edges (the robust solve).
template <bool EDGES>
__global__ void level0_kernel(const float* __restrict__ g, const float* __restrict__ conf, int w, int h, float inv, float inv2s2, int mode,
                              float lambda, float* __restrict__ ex, float* __restrict__ ey, float* __restrict__ ax, float* __restrict__ ay,
                              float* __restrict__ wd, float* __restrict__ dinv, const HOps H) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const size_t k = (size_t)y * w + x;
    const bool L = x > 0, R = x + 1 < w, T = y > 0, B = y + 1 < h;
    const float wv = __fadd_rn(fmaxf(conf[k], 0.f), 1e-4f);
    float al, ar, at, ab;
    if (EDGES) {
        const float gc = g[k];
        auto edge = [&](float a, float b) {
            const float d = fabsf(__fsub_rn(a, b));
            return mode == 0 ? expf(__fmul_rn(d, inv)) : expf(-__fmul_rn(__fmul_rn(d, d), inv2s2));
        };
        const float vx = R ? edge(gc, g[k + 1]) : 0.f, vy = B ? edge(gc, g[k + w]) : 0.f;
        al = L ? __fmul_rn(lambda, edge(g[k - 1], gc)) : 0.f;
        at = T ? __fmul_rn(lambda, edge(g[k - w], gc)) : 0.f;
        ar = __fmul_rn(lambda, vx);
        ab = __fmul_rn(lambda, vy);
        ex[k] = vx;
        ey[k] = vy;
        ax[k] = ar;
        ay[k] = ab;
    } else {
        al = L ? ax[k - 1] : 0.f;
        ar = ax[k];
        at = T ? ay[k - w] : 0.f;
        ab = ay[k];
    }
    wd[k] = wv;
    const float dv = dinv_of(wv, L, al, R, ar, T, at, B, ab);
    dinv[k] = dv;
    put_ops(H, k, wv, ar, ab, dv);
}
// depth.rs:852 `coarsen`, one coarse cell's right and lower edge from the finer level's
__device__ __forceinline__ float coarse_ax(const float* ax, int w, int h, int xx, int yy) {
    float a = 0.f;
    for (int y = 2 * yy; y < min(2 * yy + 2, h); y++) a = __fadd_rn(a, ax[(size_t)y * w + 2 * xx + 1]);
    return a;
}
__device__ __forceinline__ float coarse_ay(const float* ay, int w, int h, int xx, int yy) {
    float b = 0.f;
    for (int x = 2 * xx; x < min(2 * xx + 2, w); x++) b = __fadd_rn(b, ay[(size_t)(2 * yy + 1) * w + x]);
    return b;
}
// depth.rs:886 `coarsen_wd_into`, depth.rs:911 `restrict`: 2x2 block sums
__device__ __forceinline__ float block_sum_at(const float* src, int w, int h, int xx, int yy) {
    float o = 0.f;
    for (int y = 2 * yy; y < min(2 * yy + 2, h); y++) {
        float rs = 0.f;
        for (int x = 2 * xx; x < min(2 * xx + 2, w); x++) rs = __fadd_rn(rs, src[(size_t)y * w + x]);
        o = __fadd_rn(o, rs);
    }
    return o;
}
// One coarse cell of the hierarchy: its edges (EDGES; else those that are there), weight and diagonal from the finer level F.
template <bool EDGES>
__device__ __forceinline__ void coarse_cell(const WlsLevel& F, const WlsLevel& C, const HOps& H, int xx, int yy) {
    const size_t k = (size_t)yy * C.w + xx;
    const bool L = xx > 0, R = xx + 1 < C.w, T = yy > 0, B = yy + 1 < C.h;
    float al, ar, at, ab;
    if (EDGES) {
        al = L ? coarse_ax(F.ax, F.w, F.h, xx - 1, yy) : 0.f;
        ar = R ? coarse_ax(F.ax, F.w, F.h, xx, yy) : 0.f;
        at = T ? coarse_ay(F.ay, F.w, F.h, xx, yy - 1) : 0.f;
        ab = B ? coarse_ay(F.ay, F.w, F.h, xx, yy) : 0.f;
        C.ax[k] = ar;
        C.ay[k] = ab;
    } else {
        al = L ? C.ax[k - 1] : 0.f;
        ar = C.ax[k];
        at = T ? C.ay[k - C.w] : 0.f;
        ab = C.ay[k];
    }
    const float wv = block_sum_at(F.wd, F.w, F.h, xx, yy);
    C.wd[k] = wv;
    const float dv = dinv_of(wv, L, al, R, ar, T, at, B, ab);
    C.dinv[k] = dv;
    put_ops(H, k, wv, ar, ab, dv);
}
template <bool EDGES>
__global__ void coarse_level_kernel(const WlsLevel F, const WlsLevel C, const HOps H) {
    const int xx = blockIdx.x * blockDim.x + threadIdx.x, yy = blockIdx.y * blockDim.y + threadIdx.y;
    if (xx < C.w && yy < C.h) coarse_cell<EDGES>(F, C, H, xx, yy);
}
// The small levels, one after another in one CTA (each reads what the one before wrote, behind a block barrier).
constexpr int MG_TAIL_CELLS = 8192, MG_TAIL_MAX = 16;
struct MgSetup {
    WlsLevel lv[MG_TAIL_MAX + 1];  // the last large level, then the small ones
    HOps H[MG_TAIL_MAX + 1];
    int n;
};
template <bool EDGES>
__global__ void __launch_bounds__(1024) coarse_tail_kernel(const MgSetup T) {
    for (int l = 1; l < T.n; l++) {
        const WlsLevel& C = T.lv[l];
        for (int k = threadIdx.x; k < C.w * C.h; k += blockDim.x) coarse_cell<EDGES>(T.lv[l - 1], C, T.H[l], k % C.w, k / C.w);
        __syncthreads();
    }
}
// The level kernels walk strips: a warp takes 32 columns, of which the outer HALO on each side are only there for their
// neighbours (they belong to the warps beside it), and goes down `rows` rows, so that a cell's left and right neighbours
// come by shuffles, the upper and lower ones stay in registers, and the next row's operands are loaded while this one is
// worked on: every plane is read about once, no shared memory and no barrier. What bounds it: HBM and L2 on large
// grids, the latency of a row (about 1200 cycles, its loads) times the rows on small ones, hence fewer rows a strip there:
// on 2120 x 1416 the direction's pass takes 20 us with 16 rows (28 with 4, 26 with 32, 35 from shared-memory tiles).
struct Strip {
    int rows, nx, warps;  // rows a strip, strips side by side, strips in all
};
static Strip strip_of(int w, int h, int halo) {
    Strip S;
    S.nx = (w + 32 - 2 * halo - 1) / (32 - 2 * halo);
    S.rows = 32;  // an even number; at least 6 warps an SM scheduler where the level is large enough for that
    while (S.rows > 4 && S.nx * ((h + S.rows - 1) / S.rows) < 148 * 24) S.rows /= 2;
    S.warps = S.nx * ((h + S.rows - 1) / S.rows);
    return S;
}
static int strip_blocks(const Strip& S) { return (S.warps + 7) / 8; }
__device__ __forceinline__ float from_left(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float from_right(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }
// One row's operands of a lane's column (0 outside the grid).
struct RowOps {
    float wd, ax, ay, dinv, b;
};

// Sums over the grid of the CG's dot products (depth.rs:1037 `dot`: f64 products, each exact), taken by the kernel
// that has the factors in registers: each thread's sum, the block's in a fixed tree, its place in `part`; the last
// block to arrive adds the blocks' parts in a fixed order (the same values every run). True in that block, whose
// thread 0 then has the sums.
template <int NS>
__device__ __forceinline__ bool reduce_last(double (&v)[NS], double* part, int* ticket) {
    __shared__ double red[NS][8];
    __shared__ int last;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, wid = tid >> 5;
    auto block_sum = [&]() {  // 256 threads
#pragma unroll
        for (int q = 0; q < NS; q++)
            for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
        __syncthreads();
        if (lane == 0)
            for (int q = 0; q < NS; q++) red[q][wid] = v[q];
        __syncthreads();
        if (tid == 0)
            for (int q = 0; q < NS; q++) {
                double t = red[q][0];
                for (int i = 1; i < 8; i++) t += red[q][i];
                v[q] = t;
            }
    };
    block_sum();
    if (tid == 0) {
        for (int q = 0; q < NS; q++) part[(size_t)q * gridDim.x + blockIdx.x] = v[q];
        __threadfence();
        last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    for (int q = 0; q < NS; q++) {
        double t = 0.0;
        for (int i = tid; i < (int)gridDim.x; i += 256) t += __ldcg(part + (size_t)q * gridDim.x + i);
        v[q] = t;
    }
    block_sum();
    if (tid == 0) *ticket = 0;
    return true;
}
// The CG's scalars on the device and what the host reads.
struct CgOut {
    float rel;
    int stop, iters, pad;
    double rel64;
};
struct CgRef {
    double *part, *scal;
    float* ab;
    int* ctl;
    CgOut* host;
};
// depth.rs:1074 beta = r.z / the one before (the first direction is z), behind the preconditioner's last pass
__device__ __forceinline__ void cg_rz(const CgRef& C, double rz) {
    C.ab[1] = C.ctl[1] > 0 ? (float)(rz / C.scal[0]) : 0.f;
    C.scal[0] = rz;
}
__device__ __forceinline__ void cg_rel(const CgRef& C, double rr, int iters, bool stop) {
    const double rel = sqrt(rr) / C.scal[1];
    const float relf = (float)rel;
    stop = stop || relf < 1e-5f;
    C.ctl[0] = stop;
    C.ctl[1] = iters;
    C.host->rel = relf;
    C.host->rel64 = rel;
    C.host->iters = iters;
    C.host->stop = stop;
}
// depth.rs:1039: b = W d, r = b - A u, |b| and |r|.
__global__ void __launch_bounds__(256) cg_start_kernel(const float* __restrict__ d, const float* __restrict__ u, const float* __restrict__ wd,
                                                       const float* __restrict__ ax, const float* __restrict__ ay, float* __restrict__ r, int w,
                                                       int h, const Strip S, const CgRef C) {
    const int lane = threadIdx.x & 31, wid = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int gx = wid % S.nx * 30 + lane - 1, y0 = wid / S.nx * S.rows, y1 = wid < S.warps ? min(h, y0 + S.rows) : 0;
    const bool inx = gx >= 0 && gx < w, own = lane >= 1 && lane <= 30 && gx < w;
    auto U = [&](int y) { return inx && y >= 0 && y < h ? u[(size_t)y * w + gx] : 0.f; };
    double v[2] = {0.0, 0.0};
    if (y0 < y1) {
        float um = U(y0 - 1), uc = U(y0), aym = inx && y0 > 0 ? ay[(size_t)(y0 - 1) * w + gx] : 0.f;
#pragma unroll 2
        for (int y = y0; y < y1; y++) {
            const size_t k = (size_t)y * w + gx;
            const float un = U(y + 1), wk = inx ? wd[k] : 0.f, axk = inx ? ax[k] : 0.f, ayk = inx ? ay[k] : 0.f, dk = inx ? d[k] : 0.f;
            const float ul = from_left(uc), ur = from_right(uc), al = from_left(axk);
            if (own) {
                const float bk = __fmul_rn(wk, dk);
                float a = __fmul_rn(wk, uc);
                if (gx > 0) a = __fadd_rn(a, __fmul_rn(al, __fsub_rn(uc, ul)));
                if (gx + 1 < w) a = __fadd_rn(a, __fmul_rn(axk, __fsub_rn(uc, ur)));
                if (y > 0) a = __fadd_rn(a, __fmul_rn(aym, __fsub_rn(uc, um)));
                if (y + 1 < h) a = __fadd_rn(a, __fmul_rn(ayk, __fsub_rn(uc, un)));
                const float rv = __fsub_rn(bk, a);
                r[k] = rv;
                v[0] += (double)bk * (double)bk;
                v[1] += (double)rv * (double)rv;
            }
            um = uc;
            uc = un;
            aym = ayk;
        }
    }
    if (reduce_last(v, C.part, C.ctl + 2) && threadIdx.x == 0) {
        C.scal[1] = fmax(sqrt(v[0]), 1e-30);
        cg_rel(C, v[1], 0, false);
    }
}
// depth.rs:1074 p = z + beta p, then depth.rs:1056 A p and p.Ap -> alpha: the direction computed from z and the last one,
// which stays in the other buffer (the strips beside read it).
__global__ void __launch_bounds__(256) cg_dir_kernel(const float* __restrict__ z, float* p0, float* p1, const float* __restrict__ wd,
                                                     const float* __restrict__ ax, const float* __restrict__ ay, float* __restrict__ ap, int w,
                                                     int h, const Strip S, const CgRef C) {
    if (C.ctl[0]) return;
    const int it = C.ctl[1], lane = threadIdx.x & 31, wid = blockIdx.x * 8 + (threadIdx.x >> 5);
    const bool first = it == 0;
    const float beta = C.ab[1];
    const float* __restrict__ old = it & 1 ? p1 : p0;
    float* __restrict__ now = it & 1 ? p0 : p1;
    const int gx = wid % S.nx * 30 + lane - 1, y0 = wid / S.nx * S.rows, y1 = wid < S.warps ? min(h, y0 + S.rows) : 0;
    const bool inx = gx >= 0 && gx < w, own = lane >= 1 && lane <= 30 && gx < w;
    auto P = [&](int y) {
        if (!inx || y < 0 || y >= h) return 0.f;
        const size_t k = (size_t)y * w + gx;
        return first ? z[k] : __fadd_rn(z[k], __fmul_rn(beta, old[k]));
    };
    double v[1] = {0.0};
    if (y0 < y1) {
        float pm = P(y0 - 1), pc = P(y0), aym = inx && y0 > 0 ? ay[(size_t)(y0 - 1) * w + gx] : 0.f;
#pragma unroll 2
        for (int y = y0; y < y1; y++) {
            const size_t k = (size_t)y * w + gx;
            const float pn = P(y + 1), wk = inx ? wd[k] : 0.f, axk = inx ? ax[k] : 0.f, ayk = inx ? ay[k] : 0.f;
            const float pl = from_left(pc), pr = from_right(pc), al = from_left(axk);
            if (own) {
                float a = __fmul_rn(wk, pc);
                if (gx > 0) a = __fadd_rn(a, __fmul_rn(al, __fsub_rn(pc, pl)));
                if (gx + 1 < w) a = __fadd_rn(a, __fmul_rn(axk, __fsub_rn(pc, pr)));
                if (y > 0) a = __fadd_rn(a, __fmul_rn(aym, __fsub_rn(pc, pm)));
                if (y + 1 < h) a = __fadd_rn(a, __fmul_rn(ayk, __fsub_rn(pc, pn)));
                now[k] = pc;
                ap[k] = a;
                v[0] += (double)pc * (double)a;
            }
            pm = pc;
            pc = pn;
            aym = ayk;
        }
    }
    if (reduce_last(v, C.part, C.ctl + 2) && threadIdx.x == 0) {
        // p.Ap <= 0: alpha 0, u and r stay as they are and the iteration ends (depth.rs:1060)
        C.ab[0] = v[0] <= 0.0 ? 0.f : (float)(C.scal[0] / v[0]);
        C.ctl[3] = v[0] <= 0.0;
    }
}
// depth.rs:1064-1065: u += alpha p, r -= alpha Ap, |r| -> the residual; the end of an iteration.
__global__ void __launch_bounds__(256) cg_step_kernel(float* __restrict__ u, const float* __restrict__ p0, const float* __restrict__ p1,
                                                      float* __restrict__ r, const float* __restrict__ ap, size_t n, int max_iters, const CgRef C) {
    if (C.ctl[0]) return;  // an iteration queued ahead of the last one's result
    const float alpha = C.ab[0];
    const float* p = C.ctl[1] & 1 ? p0 : p1;
    double v[1] = {0.0};
    const size_t t0 = blockIdx.x * (size_t)256 + threadIdx.x, nt = (size_t)gridDim.x * 256;
    auto one = [&](float& uv, float pv, float& rv, float av) {
        uv = __fadd_rn(uv, __fmul_rn(alpha, pv));
        rv = __fsub_rn(rv, __fmul_rn(alpha, av));
        v[0] += (double)rv * (double)rv;
    };
    const bool vec = ((reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(r) |
                       reinterpret_cast<uintptr_t>(ap)) & 15) == 0;
    const size_t n4 = vec ? n / 4 : 0;
    for (size_t i = t0; i < n4; i += nt) {
        float4 uv = reinterpret_cast<float4*>(u)[i], rv = reinterpret_cast<float4*>(r)[i];
        const float4 pv = reinterpret_cast<const float4*>(p)[i], av = reinterpret_cast<const float4*>(ap)[i];
        one(uv.x, pv.x, rv.x, av.x);
        one(uv.y, pv.y, rv.y, av.y);
        one(uv.z, pv.z, rv.z, av.z);
        one(uv.w, pv.w, rv.w, av.w);
        reinterpret_cast<float4*>(u)[i] = uv;
        reinterpret_cast<float4*>(r)[i] = rv;
    }
    for (size_t i = 4 * n4 + t0; i < n; i += nt) one(u[i], p[i], r[i], ap[i]);
    if (reduce_last(v, C.part, C.ctl + 2) && threadIdx.x == 0) {
        const int it = C.ctl[1] + 1;
        cg_rel(C, v[0], it, C.ctl[3] != 0 || it >= max_iters);
    }
}
// r.z alone, for a preconditioner that ends in a copy (a grid small enough for one CTA).
__global__ void __launch_bounds__(256) cg_rz_kernel(const float* __restrict__ r, const float* __restrict__ z, size_t n, const CgRef C) {
    double v[1] = {0.0};
    for (size_t i = blockIdx.x * (size_t)256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) v[0] += (double)r[i] * (double)z[i];
    if (reduce_last(v, C.part, C.ctl + 2) && threadIdx.x == 0) cg_rz(C, v[0]);
}

// One fine level's way down the V-cycle in one pass (depth.rs:924-930): the zero-start Jacobi sweep x = w D^-1 b
// (depth.rs:840), the residual b - A x (depth.rs:786) and its restriction to the coarse right-hand side (depth.rs:911).
// A lane's pair of columns (even, odd) belongs to one coarse cell: the odd one's residual comes by a shuffle.
__global__ void __launch_bounds__(256) vc_down_kernel(const float* __restrict__ b, const float* __restrict__ wd, const float* __restrict__ ax,
                                                      const float* __restrict__ ay, const float* __restrict__ dinv, float* __restrict__ x,
                                                      int w, int h, float* __restrict__ cb, int cw, const Strip S) {
    const int lane = threadIdx.x & 31, wid = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (wid >= S.warps) return;
    const int gx = wid % S.nx * 30 + lane - 1, y0 = wid / S.nx * S.rows, y1 = min(h, y0 + S.rows);
    const bool inx = gx >= 0 && gx < w, own = lane >= 1 && lane <= 30 && gx < w;
    float bc = 0.f, bn = 0.f;  // b of this row and the next
    auto J = [&](int y, float& bv) {
        bv = 0.f;
        if (!inx || y < 0 || y >= h) return 0.f;
        const size_t k = (size_t)y * w + gx;
        bv = b[k];
        return __fmul_rn(__fmul_rn(MG_OMEGA, dinv[k]), bv);
    };
    float xm = J(y0 - 1, bc), xc = J(y0, bc), aym = inx && y0 > 0 ? ay[(size_t)(y0 - 1) * w + gx] : 0.f, o = 0.f;
#pragma unroll 2
    for (int y = y0; y < y1; y++) {
        const size_t k = (size_t)y * w + gx;
        const float xn = J(y + 1, bn), wk = inx ? wd[k] : 0.f, axk = inx ? ax[k] : 0.f, ayk = inx ? ay[k] : 0.f;
        const float xl = from_left(xc), xr = from_right(xc), al = from_left(axk);
        float r = 0.f;
        if (own) {
            float v = __fmul_rn(wk, xc);
            if (gx > 0) v = __fadd_rn(v, __fmul_rn(al, __fsub_rn(xc, xl)));
            if (gx + 1 < w) v = __fadd_rn(v, __fmul_rn(axk, __fsub_rn(xc, xr)));
            if (y > 0) v = __fadd_rn(v, __fmul_rn(aym, __fsub_rn(xc, xm)));
            if (y + 1 < h) v = __fadd_rn(v, __fmul_rn(ayk, __fsub_rn(xc, xn)));
            r = __fsub_rn(bc, v);
            x[k] = xc;
        }
        const float r1 = from_right(r);  // strips start at even columns and rows
        float rs = __fadd_rn(0.f, r);
        if (gx + 1 < w) rs = __fadd_rn(rs, r1);
        o = __fadd_rn(y & 1 ? o : 0.f, rs);
        if (own && !(gx & 1) && ((y & 1) || y + 1 == h)) cb[(size_t)(y >> 1) * cw + (gx >> 1)] = o;
        xm = xc;
        xc = xn;
        bc = bn;
        aym = ayk;
    }
}
// ... and its way up in one pass (depth.rs:932-946): the prolongation x += P x_c (depth.rs:901) and the damped Jacobi
// sweep (depth.rs:837) on the corrected x, into out (another buffer than x). DOT (level 0): r.z taken on the way (b is
// the CG's r).
template <bool DOT>
__global__ void __launch_bounds__(256) vc_up_kernel(const float* __restrict__ x, const float* __restrict__ xc_, int cw,
                                                    const float* __restrict__ b, const float* __restrict__ wd,
                                                    const float* __restrict__ ax, const float* __restrict__ ay,
                                                    const float* __restrict__ dinv, float* __restrict__ out, int w, int h, const Strip S,
                                                    const CgRef C) {
    if (DOT && C.ctl[0]) return;
    const int lane = threadIdx.x & 31, wid = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int gx = wid % S.nx * 30 + lane - 1, y0 = wid / S.nx * S.rows, y1 = wid < S.warps ? min(h, y0 + S.rows) : 0;
    const bool inx = gx >= 0 && gx < w, own = lane >= 1 && lane <= 30 && gx < w;
    auto X = [&](int y) { return inx && y >= 0 && y < h ? __fadd_rn(x[(size_t)y * w + gx], xc_[(size_t)(y >> 1) * cw + (gx >> 1)]) : 0.f; };
    double v[1] = {0.0};
    if (y0 < y1) {
        float xm = X(y0 - 1), xc = X(y0), aym = inx && y0 > 0 ? ay[(size_t)(y0 - 1) * w + gx] : 0.f;
#pragma unroll 2
        for (int y = y0; y < y1; y++) {
            const size_t k = (size_t)y * w + gx;
            const float xn = X(y + 1), wk = inx ? wd[k] : 0.f, axk = inx ? ax[k] : 0.f, ayk = inx ? ay[k] : 0.f, bk = inx ? b[k] : 0.f,
                        dk = inx ? dinv[k] : 0.f;
            const float xl = from_left(xc), xr = from_right(xc), al = from_left(axk);
            if (own) {
                float a = __fmul_rn(wk, xc);
                if (gx > 0) a = __fadd_rn(a, __fmul_rn(al, __fsub_rn(xc, xl)));
                if (gx + 1 < w) a = __fadd_rn(a, __fmul_rn(axk, __fsub_rn(xc, xr)));
                if (y > 0) a = __fadd_rn(a, __fmul_rn(aym, __fsub_rn(xc, xm)));
                if (y + 1 < h) a = __fadd_rn(a, __fmul_rn(ayk, __fsub_rn(xc, xn)));
                const float o = __fadd_rn(xc, __fmul_rn(__fmul_rn(MG_OMEGA, dk), __fsub_rn(bk, a)));
                out[k] = o;
                if (DOT) v[0] += (double)bk * (double)o;
            }
            xm = xc;
            xc = xn;
            aym = ayk;
        }
    }
    if (DOT && reduce_last(v, C.part, C.ctl + 2) && threadIdx.x == 0) cg_rz(C, v[0]);
}

__device__ __forceinline__ void cp_async4f(float* smem, const float* gmem) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// The coarse end of the V-cycle (depth.rs:924 `vcycle` from level 0 of `T` down) in ONE CTA: each level's zero-start
// Jacobi, residual and restriction, the coarsest level's MG_COARSE sweeps, then prolongation and the smoothing sweep
// back up. The per-element arithmetic is the separate kernels'. The levels' x and b live in shared memory, and below
// the first level their operators too (copied while the first level is worked on); the coarsest level (at most 256
// cells) is one cell per thread with its operators in registers and x in two shared buffers, one barrier a sweep.
// What bounds it: latency, barrier by barrier (MG_COARSE of its about 45 are the sweeps'). With everything in global
// memory and two barriers a sweep it took 22 to 27 us of an iteration, 14 to 20 here (one SM's instruction rate).
struct MgTail {
    WlsLevel lv[MG_TAIL_MAX];
    int n;
};
constexpr int TAIL_THREADS = 1024, TAIL_PER = MG_TAIL_CELLS / TAIL_THREADS;
// floats of shared memory: x and b of every level, the operators (wd, ax, ay, dinv) below the first, a spare x for the coarsest
static size_t tail_floats(const WlsSolver* S, size_t l) {
    size_t f = 256;
    for (size_t q = l; q < S->lv.size(); q++) f += (size_t)S->lv[q].w * S->lv[q].h * (q == l ? 2 : 6);
    return f;
}
constexpr size_t TAIL_MAX_SMEM = 220 * 1024;
struct TailOps {  // a level's operators and vectors as the tail reads them
    const float *wd, *ax, *ay, *dinv;
    float *x, *b;
    int w, h;
};
// A x of one cell: the neighbours from x, in the order left, right, up, down (depth.rs:786)
__device__ __forceinline__ float tail_apply(const TailOps& L, int k, int i, int y) {
    const float xk = L.x[k];
    float v = __fmul_rn(L.wd[k], xk);
    if (i > 0) v = __fadd_rn(v, __fmul_rn(L.ax[k - 1], __fsub_rn(xk, L.x[k - 1])));
    if (i + 1 < L.w) v = __fadd_rn(v, __fmul_rn(L.ax[k], __fsub_rn(xk, L.x[k + 1])));
    if (y > 0) v = __fadd_rn(v, __fmul_rn(L.ay[k - L.w], __fsub_rn(xk, L.x[k - L.w])));
    if (y + 1 < L.h) v = __fadd_rn(v, __fmul_rn(L.ay[k], __fsub_rn(xk, L.x[k + L.w])));
    return v;
}
__global__ void __launch_bounds__(TAIL_THREADS) vcycle_tail_kernel(const MgTail T) {
    extern __shared__ float tail_sm[];
    const int tid = threadIdx.x;
    // where level l lies (the few levels are walked again by every thread: no table to wait for)
    auto level = [&](int l) {
        float* at = tail_sm + 256;
        TailOps L{};
        for (int q = 0; q <= l; q++) {
            const WlsLevel& G = T.lv[q];
            const int n = G.w * G.h;
            L.w = G.w;
            L.h = G.h;
            L.x = at;
            L.b = at + n;
            if (q == 0) {
                L.wd = G.wd, L.ax = G.ax, L.ay = G.ay, L.dinv = G.dinv;
                at += 2 * n;
            } else {
                L.wd = at + 2 * n, L.ax = at + 3 * n, L.ay = at + 4 * n, L.dinv = at + 5 * n;
                at += 6 * n;
            }
        }
        return L;
    };
    // the operators below the first level, on their way while it is worked on
    for (int l = 1; l < T.n; l++) {
        const WlsLevel& G = T.lv[l];
        const TailOps L = level(l);
        const int n = G.w * G.h;
        for (int k = tid; k < n; k += TAIL_THREADS) {
            cp_async4f(const_cast<float*>(L.wd) + k, G.wd + k);
            cp_async4f(const_cast<float*>(L.ax) + k, G.ax + k);
            cp_async4f(const_cast<float*>(L.ay) + k, G.ay + k);
            cp_async4f(const_cast<float*>(L.dinv) + k, G.dinv + k);
        }
    }
    cp_commit();
    for (int l = 0; l + 1 < T.n; l++) {
        const TailOps L = level(l), C = level(l + 1);
        const int n = L.w * L.h;
        if (l == 0)
            for (int k = tid; k < n; k += TAIL_THREADS) L.b[k] = T.lv[0].b[k];
        for (int k = tid; k < n; k += TAIL_THREADS) L.x[k] = __fmul_rn(__fmul_rn(MG_OMEGA, L.dinv[k]), L.b[k]);
        __syncthreads();
        // the residual's 2x2 block sums, a coarse cell per thread
        for (int k = tid; k < C.w * C.h; k += TAIL_THREADS) {
            const int xx = k % C.w, yy = k / C.w;
            float o = 0.f;
            for (int y = 2 * yy; y < min(2 * yy + 2, L.h); y++) {
                float rs = 0.f;
                for (int x = 2 * xx; x < min(2 * xx + 2, L.w); x++) {
                    const int q = y * L.w + x;
                    rs = __fadd_rn(rs, __fsub_rn(L.b[q], tail_apply(L, q, x, y)));
                }
                o = __fadd_rn(o, rs);
            }
            C.b[k] = o;
        }
        if (l == 0) cp_wait<0>();
        __syncthreads();
    }
    {
        const TailOps Z = level(T.n - 1);
        const int n = Z.w * Z.h;
        if (T.n == 1) {
            for (int k = tid; k < n; k += TAIL_THREADS) Z.b[k] = T.lv[0].b[k];
            __syncthreads();
        }
        const bool mine = tid < n;  // the coarsest level: at most MG_MIN x MG_MIN = 256 cells
        const int i = tid % Z.w, y = tid / Z.w;
        const bool l = mine && i > 0, r = mine && i + 1 < Z.w, t = mine && y > 0, b = mine && y + 1 < Z.h;
        const float wk = mine ? Z.wd[tid] : 0.f, od = mine ? __fmul_rn(MG_OMEGA, Z.dinv[tid]) : 0.f, bk = mine ? Z.b[tid] : 0.f;
        const float al = l ? Z.ax[tid - 1] : 0.f, ar = r ? Z.ax[tid] : 0.f, at = t ? Z.ay[tid - Z.w] : 0.f, ab = b ? Z.ay[tid] : 0.f;
        float *src = tail_sm, *dst = Z.x;  // MG_COARSE even: the last sweep writes Z.x
        float xk = __fmul_rn(od, bk);
        if (mine) src[tid] = xk;
        if (tid < 256) {
            for (int it = 1; it < MG_COARSE; it++) {
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (mine) {
                    float v = __fmul_rn(wk, xk);
                    if (l) v = __fadd_rn(v, __fmul_rn(al, __fsub_rn(xk, src[tid - 1])));
                    if (r) v = __fadd_rn(v, __fmul_rn(ar, __fsub_rn(xk, src[tid + 1])));
                    if (t) v = __fadd_rn(v, __fmul_rn(at, __fsub_rn(xk, src[tid - Z.w])));
                    if (b) v = __fadd_rn(v, __fmul_rn(ab, __fsub_rn(xk, src[tid + Z.w])));
                    xk = __fadd_rn(xk, __fmul_rn(od, __fsub_rn(bk, v)));
                    dst[tid] = xk;
                }
                float* q = src;
                src = dst;
                dst = q;
            }
        }
        __syncthreads();
    }
    static_assert(MG_COARSE % 2 == 0, "the last sweep is written to Z.x");
    for (int l = T.n - 2; l >= 0; l--) {
        const TailOps L = level(l), C = level(l + 1);
        const int n = L.w * L.h;
        for (int k = tid; k < n; k += TAIL_THREADS) {
            const int i = k % L.w, y = k / L.w;
            L.x[k] = __fadd_rn(L.x[k], C.x[(y / 2) * C.w + i / 2]);
        }
        __syncthreads();
        float nv[TAIL_PER];
#pragma unroll
        for (int q = 0; q < TAIL_PER; q++) {
            const int k = tid + q * TAIL_THREADS;
            if (k < n) nv[q] = __fadd_rn(L.x[k], __fmul_rn(__fmul_rn(MG_OMEGA, L.dinv[k]), __fsub_rn(L.b[k], tail_apply(L, k, k % L.w, k / L.w))));
        }
        if (l > 0) __syncthreads();
        float* out = l > 0 ? L.x : T.lv[0].x;
#pragma unroll
        for (int q = 0; q < TAIL_PER; q++)
            if (tid + q * TAIL_THREADS < n) out[tid + q * TAIL_THREADS] = nv[q];
        __syncthreads();
    }
    if (T.n == 1) {
        const TailOps Z = level(0);
        for (int k = tid; k < Z.w * Z.h; k += TAIL_THREADS) T.lv[0].x[k] = Z.x[k];
    }
}

// depth.rs:677 `solve_rows` / :707 `solve_cols`: the Thomas algorithm along
// every line, one thread per line, 32 lines per warp. The warp stages 32x32
// tiles of the coefficients through shared memory with coalesced row-segment
// loads (ROWS: a line is an image row, the tile is [line][element]; else a
// line is a column, the tile is [element][line]); each thread then walks its
// line's 32 elements of the tile in the reference's order and arithmetic.
constexpr int TT = 32;
template <bool ROWS>
__device__ __forceinline__ float& tl(float (*t)[TT + 1], int line, int e) {
    return ROWS ? t[line][e] : t[e][line];
}
// The 32 lines' elements e0 .. e0+31 of `src` into tile t (cp.async; `fill` where out of range).
template <bool ROWS>
__device__ __forceinline__ void tile_load(float (*t)[TT + 1], const float* __restrict__ src, int l0, int e0, int nlines, int len, int w,
                                          float fill) {
    const int lane = threadIdx.x;
    for (int q = 0; q < TT; q++) {
        const int ln = ROWS ? q : lane, e = ROWS ? e0 + lane : e0 + q;
        float* d = &tl<ROWS>(t, ln, e - e0);
        if (l0 + ln < nlines && e < len) cp_async4f(d, src + (ROWS ? (size_t)(l0 + ln) * w + e : (size_t)e * w + (l0 + ln)));
        else *d = fill;
    }
}
template <bool ROWS>
__device__ __forceinline__ void tile_store(float (*t)[TT + 1], float* __restrict__ dst, int l0, int e0, int nlines, int len, int w) {
    const int lane = threadIdx.x;
    for (int q = 0; q < TT; q++) {
        const int ln = ROWS ? q : lane, e = ROWS ? e0 + lane : e0 + q;
        if (l0 + ln < nlines && e < len) dst[ROWS ? (size_t)(l0 + ln) * w + e : (size_t)e * w + (l0 + ln)] = tl<ROWS>(t, ln, e - e0);
    }
}

// depth.rs:677 `solve_rows` / :707 `solve_cols`: the Thomas algorithm along
// every line, one thread per line, 32 lines per warp (ROWS: a line is an image
// row, the tile is [line][element]; else a line is a column, the tile is
// [element][line]). The coefficient tiles of the next 32 elements stream into
// shared memory (cp.async, two buffers) while the current 32 are eliminated,
// and the back substitution streams cp / dp the same way; each thread walks
// its line in the reference's order and arithmetic.
template <bool ROWS>
__global__ void __launch_bounds__(32) thomas_kernel(float* __restrict__ u, const float* __restrict__ f, const float* __restrict__ wd,
                                                    int unit_wd, const float* __restrict__ a, int w, int h, float lam,
                                                    float* __restrict__ cp, float* __restrict__ dp) {
    __shared__ float ta[2][TT][TT + 1], tw[2][TT][TT + 1], tf[2][TT][TT + 1], tc[2][TT][TT + 1], td[2][TT][TT + 1];
    const int lane = threadIdx.x;
    const int nlines = ROWS ? h : w, len = ROWS ? w : h;
    const int l0 = blockIdx.x * TT;
    const int li = l0 + lane;
    const int nch = (len + TT - 1) / TT;
    auto issue_fwd = [&](int c) {
        const int b = c & 1, e0 = c * TT;
        tile_load<ROWS>(ta[b], a, l0, e0, nlines, len, w, 0.f);
        tile_load<ROWS>(tf[b], f, l0, e0, nlines, len, w, 0.f);
        if (!unit_wd) tile_load<ROWS>(tw[b], wd, l0, e0, nlines, len, w, 1.f);
        cp_commit();
    };
    float prev_a = 0.f, cprev = 0.f, dprev = 0.f;
    const float nl = -lam;
    issue_fwd(0);
    for (int c = 0; c < nch; c++) {
        const int b = c & 1, e0 = c * TT, ne = min(TT, len - e0);
        if (c + 1 < nch) {
            issue_fwd(c + 1);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncwarp();
        if (li < nlines)
            for (int j = 0; j < ne; j++) {
                const int i = e0 + j;
                const float ai = i + 1 < len ? tl<ROWS>(ta[b], lane, j) : 0.f;
                const float wdi = unit_wd ? 1.f : tl<ROWS>(tw[b], lane, j);
                const float diag = __fadd_rn(wdi, __fmul_rn(lam, __fadd_rn(prev_a, ai)));
                const float lower = __fmul_rn(nl, prev_a), upper = __fmul_rn(nl, ai);
                float m = __fsub_rn(diag, __fmul_rn(lower, i > 0 ? cprev : 0.f));
                if (fabsf(m) < 1e-12f) m = 1e-12f;
                cprev = __fdiv_rn(upper, m);
                dprev = __fdiv_rn(__fsub_rn(__fmul_rn(wdi, tl<ROWS>(tf[b], lane, j)), __fmul_rn(lower, i > 0 ? dprev : 0.f)), m);
                tl<ROWS>(tc[b], lane, j) = cprev;
                tl<ROWS>(td[b], lane, j) = dprev;
                prev_a = ai;
            }
        __syncwarp();
        if (c + 1 < nch) {  // the last chunk stays in shared memory for the back substitution
            tile_store<ROWS>(tc[b], cp, l0, e0, nlines, len, w);
            tile_store<ROWS>(td[b], dp, l0, e0, nlines, len, w);
        }
        __syncwarp();
    }
    __threadfence_block();
    __syncwarp();
    // back substitution, chunks from the end; chunk c-1's cp / dp stream in while chunk c runs
    const int last = nch - 1;
    auto issue_bwd = [&](int c) {
        const int b = c & 1, e0 = c * TT;
        tile_load<ROWS>(tc[b], cp, l0, e0, nlines, len, w, 0.f);
        tile_load<ROWS>(td[b], dp, l0, e0, nlines, len, w, 0.f);
        cp_commit();
    };
    float nxt = 0.f;
    for (int c = last; c >= 0; c--) {
        const int b = c & 1, e0 = c * TT, ne = min(TT, len - e0);
        if (c - 1 >= 0) {
            issue_bwd(c - 1);
            if (c != last) cp_wait<1>();
        } else if (c != last) {
            cp_wait<0>();
        }
        __syncwarp();
        if (li < nlines)
            for (int j = ne - 1; j >= 0; j--) {
                const int i = e0 + j;
                nxt = i == len - 1 ? tl<ROWS>(td[b], lane, j) : __fsub_rn(tl<ROWS>(td[b], lane, j), __fmul_rn(tl<ROWS>(tc[b], lane, j), nxt));
                tl<ROWS>(tf[b], lane, j) = nxt;
            }
        __syncwarp();
        tile_store<ROWS>(tf[b], u, l0, e0, nlines, len, w);
        __syncwarp();
    }
    cp_wait<0>();
}
// The same systems (depth.rs:677 / :707), each line cut into P segments
// (the partition method); a warp per segment holds 32 lines (lane = line).
// (1) Each segment eliminates forward (pivots d', the spike g on the unknown
// before the segment, the right-hand side r') and backward, leaving each of
// its unknowns as rho + sigma * X_{s-1} + tau * X_s, X_s being the segment's
// last unknown. (2) One thread per line solves the P-unknown tridiagonal
// system that the segments' last equations make of the X_s. (3) Each segment
// recovers its unknowns. A line's sequential chain shrinks P-fold and P times
// as many threads run the lines; the result differs from the one-thread
// Thomas sweep by rounding only (the systems are diagonally dominant), and
// these sweeps only start the MG-PCG solve.
template <bool ROWS, int P>
__global__ void __launch_bounds__(32 * P) pthomas_kernel(float* __restrict__ u, const float* __restrict__ f, const float* __restrict__ wd,
                                                         int unit_wd, const float* __restrict__ a, int w, int h, float lam,
                                                         float* __restrict__ s0, float* __restrict__ s1, float* __restrict__ s2) {
    __shared__ float cf[P][7][32];  // per segment and line: the first unknown's (rho, sigma, tau); the last equation's d', g, r', u
    __shared__ float X[P][32];      // the segments' last unknowns
    __shared__ float rc[P][32], rr[P][32];
    const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
    const int nlines = ROWS ? h : w, len = ROWS ? w : h;
    const int line = blockIdx.x * 32 + lane;
    const bool live = line < nlines;
    const int b = (int)((long long)seg * len / P), e = (int)((long long)(seg + 1) * len / P);  // len >= P: never empty
    auto at = [&](int i) -> size_t { return ROWS ? (size_t)line * w + i : (size_t)i * w + line; };
    const float nl = -lam;
    if (live) {
        float a_prev = b > 0 ? a[at(b - 1)] : 0.f;
        float dprev = 1.f, gprev = 0.f, rprev = 0.f, uprev = 0.f;
        for (int i = b; i < e; i++) {
            const size_t k = at(i);
            const float ai = i + 1 < len ? a[k] : 0.f;
            const float wdi = unit_wd ? 1.f : wd[k];
            const float diag = wdi + lam * (a_prev + ai);
            const float lower = nl * a_prev, upper = nl * ai;
            const float ri = wdi * f[k];
            float dd = diag, gg = lower, rv = ri;
            if (i > b) {
                const float mlt = lower / dprev;
                dd = diag - mlt * uprev;
                gg = -(mlt * gprev);
                rv = ri - mlt * rprev;
            }
            if (fabsf(dd) < 1e-12f) dd = 1e-12f;
            s0[k] = dd;
            s1[k] = gg;
            s2[k] = rv;
            dprev = dd;
            gprev = gg;
            rprev = rv;
            uprev = upper;
            a_prev = ai;
        }
        cf[seg][3][lane] = dprev;
        cf[seg][4][lane] = gprev;
        cf[seg][5][lane] = rprev;
        cf[seg][6][lane] = uprev;
        float rn = 0.f, sn = 0.f, tn = 1.f;  // the last unknown is X_s itself
        {
            const size_t k = at(e - 1);
            s0[k] = 0.f;
            s1[k] = 0.f;
            s2[k] = 1.f;
        }
        for (int i = e - 2; i >= b; i--) {
            const size_t k = at(i);
            const float upper = nl * a[k];  // i + 1 < len here
            const float inv = 1.f / s0[k];
            const float rho = (s2[k] - upper * rn) * inv, sig = (-s1[k] - upper * sn) * inv, tau = -(upper * tn) * inv;
            s0[k] = rho;
            s1[k] = sig;
            s2[k] = tau;
            rn = rho;
            sn = sig;
            tn = tau;
        }
        cf[seg][0][lane] = rn;
        cf[seg][1][lane] = sn;
        cf[seg][2][lane] = tn;
    }
    __syncthreads();
    if (seg == 0 && live) {
        // segment q's last equation: g X_{q-1} + d' X_q + u x_first(q+1) = r', x_first(q+1) = rho + sigma X_q + tau X_{q+1}
        float cprev = 0.f, rprev2 = 0.f;
        for (int q = 0; q < P; q++) {
            const bool nx = q + 1 < P;
            const float uq = cf[q][6][lane];
            const float A = q > 0 ? cf[q][4][lane] : 0.f;
            const float B = nx ? cf[q][3][lane] + uq * cf[q + 1][1][lane] : cf[q][3][lane];
            const float C = nx ? uq * cf[q + 1][2][lane] : 0.f;
            const float R = nx ? cf[q][5][lane] - uq * cf[q + 1][0][lane] : cf[q][5][lane];
            float den = B - A * cprev;
            if (fabsf(den) < 1e-12f) den = 1e-12f;
            cprev = C / den;
            rprev2 = (R - A * rprev2) / den;
            rc[q][lane] = cprev;
            rr[q][lane] = rprev2;
        }
        float xn = 0.f;
        for (int q = P - 1; q >= 0; q--) {
            xn = q == P - 1 ? rr[q][lane] : rr[q][lane] - rc[q][lane] * xn;
            X[q][lane] = xn;
        }
    }
    __syncthreads();
    if (live) {
        const float xl = seg > 0 ? X[seg - 1][lane] : 0.f, xs = X[seg][lane];
        for (int i = b; i < e; i++) {
            const size_t k = at(i);
            u[k] = s0[k] + s1[k] * xl + s2[k] * xs;
        }
    }
}
constexpr int PT_ROWS = 8, PT_COLS = 16;

// The same partition method with a line's data in shared memory and many short segments (up to 128 a line): a
// CTA holds LC lines (rows: one; columns: up to 8, a 32-byte sector of each image row), thread = (segment, line),
// segments of `ept` elements (odd: conflict-free). (1) Each segment eliminates forward to its last equation
// g X_{s-1} + d X_s + u x_next = r, and backward to its first unknown x_b = rho + sig X_{s-1} + tau X_s. (2) The
// segments' last unknowns X_s form a tridiagonal system, solved by parallel cyclic reduction across the threads
// (log2 steps; the system is diagonally dominant, as the line's is). (3) With X_{s-1} and X_s known each segment
// solves its unknowns in place. Elements past the line's end are decoupled unknowns (a = 0, weight 1, right-hand
// side 0), so that every segment is whole.
// What bounds it: the divisions' latency along a segment (three a cell) and one read and one write of each plane;
// the earlier forms walked 32 segments of a row per warp, or 16 of a column through global memory, 17 words a cell:
// 0.46 and 0.38 ms a sweep on 4128 x 2752, 0.08 to 0.11 and 0.135 here.
constexpr int PTRI_SEGS = 128;
__host__ __device__ constexpr size_t ptri_smem(int segs, int ept, int lc, bool unit) {
    return sizeof(float) * ((size_t)segs * ept * lc * (unit ? 2 : 3) + (size_t)4 * segs * lc);
}
template <bool ROWS, bool UNIT, int lc>
__global__ void __launch_bounds__(ROWS ? 128 : 1024) ptri_kernel(float* __restrict__ u, const float* __restrict__ f, const float* __restrict__ wd,
                                                                 const float* __restrict__ a, int w, int h, float lam, int segs, int ept) {
    extern __shared__ float ptri_sm[];
    const int nlines = ROWS ? h : w, len = ROWS ? w : h, cells = segs * ept * lc, nt = segs * lc;
    float* A = ptri_sm;          // a, then the backward elimination's x_{i-1} coefficients
    float* F = A + cells;        // the right-hand side, then the solution
    float* WD = F + cells;       // weights (UNIT: none)
    float* red = UNIT ? WD : WD + cells;  // [4][segs][lc]
    const int tid = threadIdx.x, l0 = blockIdx.x * lc, col = tid % lc, seg = tid / lc;
    // this thread's elements of the load and the store: line l0 + col, from element seg on, segs apart (w h < 2^31)
    const bool mine = l0 + col < nlines;
    const unsigned k0 = ROWS ? (unsigned)l0 * w + seg : (unsigned)seg * w + l0 + col, dk = ROWS ? segs : (unsigned)segs * w;
    {
        unsigned k = k0;
#pragma unroll 4
        for (int i = seg, e = tid; i < segs * ept; i += segs, e += nt, k += dk) {
            const bool in = mine && i < len;
            A[e] = in && i + 1 < len ? a[k] : 0.f;
            const float wv = UNIT ? 1.f : (in ? wd[k] : 1.f), fv = in ? f[k] : 0.f;
            F[e] = UNIT ? fv : wv * fv;
            if (!UNIT) WD[e] = wv;
        }
    }
    __syncthreads();
    const float nl = -lam;
    const int base = seg * ept * lc + col;  // element j of the segment: base + j lc
    const float a_before = seg > 0 ? A[base - lc] : 0.f;
    auto guard = [](float d) { return fabsf(d) < 1e-12f ? 1e-12f : d; };
    // (1) forward: the segment's last equation
    float dp = 1.f, gp = 0.f, rp = 0.f, up = 0.f, ap = a_before;
#pragma unroll 2
    for (int j = 0; j < ept; j++) {
        const int k = base + j * lc;
        const float ai = A[k], wi = UNIT ? 1.f : WD[k], ri = F[k];
        const float diag = wi + lam * (ap + ai), lower = nl * ap;
        const float mlt = j > 0 ? lower * (1.f / dp) : 0.f;
        gp = j > 0 ? -(mlt * gp) : lower;
        rp = ri - mlt * rp;
        dp = guard(diag - mlt * up);
        up = nl * ai;
        ap = ai;
    }
    // ... and backward: its first unknown
    float P = 0.f, Q = 1.f, T = 0.f;
    {
        float ai = ept > 1 ? A[base + (ept - 2) * lc] : 0.f;
#pragma unroll 2
        for (int j = ept - 2; j >= 0; j--) {
            const int k = base + j * lc;
            const float al = j > 0 ? A[k - lc] : a_before, wi = UNIT ? 1.f : WD[k], ri = F[k];
            const float upper = nl * ai, lower = nl * al;
            const float inv = 1.f / guard(wi + lam * (al + ai) + upper * T);
            P = (ri - upper * P) * inv;
            Q = -(upper * Q) * inv;
            T = -lower * inv;
            ai = al;
        }
    }
    // (2) the reduced system
    auto R = [&](int q, int sg) -> float& { return red[(q * segs + sg) * lc + col]; };
    R(0, seg) = P;
    R(1, seg) = T;
    R(2, seg) = Q;
    __syncthreads();
    const bool nx = seg + 1 < segs;
    const float nP = nx ? R(0, seg + 1) : 0.f, nS = nx ? R(1, seg + 1) : 0.f, nT = nx ? R(2, seg + 1) : 0.f;
    float ra = gp, rb = guard(dp + up * nS), rc = up * nT, rr = rp - up * nP;
    for (int d = 1; d < segs; d *= 2) {
        __syncthreads();
        R(0, seg) = ra;
        R(1, seg) = rb;
        R(2, seg) = rc;
        R(3, seg) = rr;
        __syncthreads();
        const int lo = seg - d, hi = seg + d;
        float na = 0.f, nc = 0.f, b2 = rb, r2 = rr;
        if (lo >= 0) {
            const float q = ra * (1.f / R(1, lo));
            b2 -= R(2, lo) * q;
            r2 -= R(3, lo) * q;
            na = -(R(0, lo) * q);
        }
        if (hi < segs) {
            const float q = rc * (1.f / R(1, hi));
            b2 -= R(0, hi) * q;
            r2 -= R(3, hi) * q;
            nc = -(R(2, hi) * q);
        }
        ra = na;
        rb = guard(b2);
        rc = nc;
        rr = r2;
    }
    __syncthreads();
    const float xs = rr / rb;
    R(0, seg) = xs;
    __syncthreads();
    // (3) the segment's unknowns between X_{s-1} and X_s
    {
        float y = xs, ai = ept > 1 ? A[base + (ept - 2) * lc] : 0.f;
        T = 0.f;
        for (int j = ept - 2; j >= 0; j--) {
            const int k = base + j * lc;
            const float al = j > 0 ? A[k - lc] : a_before, wi = UNIT ? 1.f : WD[k], ri = F[k];
            const float upper = nl * ai, lower = nl * al;
            const float inv = 1.f / guard(wi + lam * (al + ai) + upper * T);
            y = (ri - upper * y) * inv;
            T = -lower * inv;
            F[k] = y;
            A[k] = T;
            ai = al;
        }
        F[base + (ept - 1) * lc] = xs;
        float x = seg > 0 ? R(0, seg - 1) : 0.f;
#pragma unroll 2
        for (int j = 0; j + 1 < ept; j++) {
            const int k = base + j * lc;
            x = F[k] + A[k] * x;
            F[k] = x;
        }
    }
    __syncthreads();
    unsigned k = k0;
#pragma unroll 4
    for (int i = seg, e = tid; i < len; i += segs, e += nt, k += dk)
        if (mine) u[k] = F[e];
}
// The sweep's shape for lines of `len`: as many segments as give them about 8 elements, 32 to 128; columns by 8, or by
// fewer where 8 do not fit shared memory. False: no shape fits (a line longer than the shared memory).
constexpr size_t PTRI_MAX_SMEM = 220 * 1024;
static bool ptri_shape(bool rows, bool unit, int len, int& lc, int& segs, int& ept) {
    segs = 32;
    while (segs < PTRI_SEGS && len > segs * 8) segs *= 2;
    ept = ((len + segs - 1) / segs) | 1;
    for (lc = rows ? 1 : 8; lc >= 1; lc /= 2)
        if (ptri_smem(segs, ept, lc, unit) <= PTRI_MAX_SMEM) return true;
    return false;
}

// One sweep of the start (weighted rows, unweighted rows or columns: the first sweep alone is weighted, and its columns are not).
// cp, dp, sc: scratch of the one-thread kernel and the global-memory partition.
static cudaError_t thomas(bool rows, float* u, const float* f, const float* wd, int unit_wd, const float* a, int w, int h, float lam,
                          float* cp, float* dp, float* sc, cudaStream_t s) {
    const int nlines = rows ? h : w, len = rows ? w : h;
    int lc, segs, ept;
    if (len >= 64 && ptri_shape(rows, unit_wd != 0, len, lc, segs, ept)) {
        const size_t smem = ptri_smem(segs, ept, lc, unit_wd != 0);
        auto go = [&](auto kern) {
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PTRI_MAX_SMEM);
            if (e != cudaSuccess) return e;
            lsb_launched(), kern<<<(nlines + lc - 1) / lc, segs * lc, smem, s>>>(u, f, wd, a, w, h, lam, segs, ept);
            return cudaGetLastError();
        };
        if (rows) return unit_wd ? go(ptri_kernel<true, true, 1>) : go(ptri_kernel<true, false, 1>);
        return lc == 8 ? go(ptri_kernel<false, true, 8>) : lc == 4 ? go(ptri_kernel<false, true, 4>)
               : lc == 2 ? go(ptri_kernel<false, true, 2>) : go(ptri_kernel<false, true, 1>);
    }
    if (len >= (rows ? PT_ROWS : PT_COLS) * 8) {
        const int g = (nlines + 31) / 32;
        if (rows) lsb_launched(), pthomas_kernel<true, PT_ROWS><<<g, 32 * PT_ROWS, 0, s>>>(u, f, wd, unit_wd, a, w, h, lam, cp, dp, sc);
        else lsb_launched(), pthomas_kernel<false, PT_COLS><<<g, 32 * PT_COLS, 0, s>>>(u, f, wd, unit_wd, a, w, h, lam, cp, dp, sc);
        return cudaGetLastError();
    }
    if (rows) lsb_launched(), thomas_kernel<true><<<(nlines + TT - 1) / TT, TT, 0, s>>>(u, f, wd, unit_wd, a, w, h, lam, cp, dp);
    else lsb_launched(), thomas_kernel<false><<<(nlines + TT - 1) / TT, TT, 0, s>>>(u, f, wd, unit_wd, a, w, h, lam, cp, dp);
    return cudaGetLastError();
}

// ------------------------------------------------ the BF16 V-cycle (mode 1)
// The preconditioner's smoother, residual, restriction and prolongation on
// BF16 copies of the level operators and vectors, arithmetic in FP32; the
// outer CG stays FP32 with FP64 dot products. No reference counterpart: the
// reference's V-cycle is FP32 (vcycle_mode 0 here).
__global__ void to_bf16_kernel(const float* __restrict__ a, uint16_t* __restrict__ o, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) sth(o, i, a[i]);
}
__global__ void from_bf16_kernel(const uint16_t* __restrict__ a, float* __restrict__ o, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) o[i] = ldh(a, i);
}
// A level's right-hand side and a sweep's output are BF16 (uint16_t) below level 0; at level 0 the
// right-hand side is the CG's FP32 residual and the last sweep writes the FP32 z.
__device__ __forceinline__ float ldv(const uint16_t* p, size_t k) { return ldh(p, k); }
__device__ __forceinline__ float ldv(const float* p, size_t k) { return p[k]; }
__device__ __forceinline__ void stv(uint16_t* p, size_t k, float v) { sth(p, k, v); }
__device__ __forceinline__ void stv(float* p, size_t k, float v) { p[k] = v; }
__device__ __forceinline__ float stencil_h_at(const uint16_t* __restrict__ x, float bk, const uint16_t* __restrict__ wd,
                                              const uint16_t* __restrict__ ax, const uint16_t* __restrict__ ay,
                                              const uint16_t* __restrict__ dinv, int w, int h, int i, int y, int mode) {
    const size_t k = (size_t)y * w + i;
    const float xk = ldh(x, k);
    float v = ldh(wd, k) * xk;
    if (i > 0) v += ldh(ax, k - 1) * (xk - ldh(x, k - 1));
    if (i + 1 < w) v += ldh(ax, k) * (xk - ldh(x, k + 1));
    if (y > 0) v += ldh(ay, k - w) * (xk - ldh(x, k - w));
    if (y + 1 < h) v += ldh(ay, k) * (xk - ldh(x, k + w));
    const float r = bk - v;
    return mode == 1 ? r : xk + MG_OMEGA * ldh(dinv, k) * r;
}
// mode 1: out = b - A x; mode 2: out = x + w D^-1 (b - A x)
template <class BT, class OT>
__global__ void stencil_h_kernel(const uint16_t* __restrict__ x, const BT* __restrict__ b, const uint16_t* __restrict__ wd,
                                 const uint16_t* __restrict__ ax, const uint16_t* __restrict__ ay, const uint16_t* __restrict__ dinv,
                                 OT* __restrict__ out, int w, int h, int mode) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= w || y >= h) return;
    const size_t k = (size_t)y * w + i;
    stv(out, k, stencil_h_at(x, ldv(b, k), wd, ax, ay, dinv, w, h, i, y, mode));
}
template <class BT>
__global__ void jac0_h_kernel(const BT* __restrict__ b, const uint16_t* __restrict__ dinv, uint16_t* __restrict__ x, size_t n) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
        sth(x, k, MG_OMEGA * ldh(dinv, k) * ldv(b, k));
}
// A fine level's way down and way up in one pass each, the values the separate sweeps would store (each rounded to
// BF16): two sweeps deep, so two halo columns a side, and each step of the walk works on three rows -- the sweep's
// start on row t, one sweep on row t - 1, the next (or the residual) on row t - 2.
__device__ __forceinline__ float rbf(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
template <class BT>
__device__ __forceinline__ RowOps row_ops(const BT* __restrict__ b, const uint16_t* __restrict__ wd, const uint16_t* __restrict__ ax,
                                          const uint16_t* __restrict__ ay, const uint16_t* __restrict__ dinv, bool in, size_t k) {
    if (!in) return RowOps{0.f, 0.f, 0.f, 0.f, 0.f};
    return RowOps{ldh(wd, k), ldh(ax, k), ldh(ay, k), ldh(dinv, k), ldv(b, k)};
}
// b - A x of a cell (its left edge al, its upper edge at; neighbours outside the grid left out)
__device__ __forceinline__ float resid_h(const RowOps& q, float al, float at, float xc, float xl, float xr, float xm, float xn, int gx, int y, int w,
                                         int h) {
    float v = q.wd * xc;
    if (gx > 0) v += al * (xc - xl);
    if (gx + 1 < w) v += q.ax * (xc - xr);
    if (y > 0) v += at * (xc - xm);
    if (y + 1 < h) v += q.ay * (xc - xn);
    return q.b - v;
}
// Down: x0 = w D^-1 b, x1 = one sweep, r = b - A x1, its 2x2 block sums; x1 -> x, the sums -> cb.
template <class BT>
__global__ void __launch_bounds__(256) vc_down_h_kernel(const BT* __restrict__ b, const uint16_t* __restrict__ wd,
                                                        const uint16_t* __restrict__ ax, const uint16_t* __restrict__ ay,
                                                        const uint16_t* __restrict__ dinv, uint16_t* __restrict__ x, int w, int h,
                                                        uint16_t* __restrict__ cb, int cw, const Strip S) {
    const int lane = threadIdx.x & 31, wid = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (wid >= S.warps) return;
    const int gx = wid % S.nx * 28 + lane - 2, y0 = wid / S.nx * S.rows, y1 = min(h, y0 + S.rows);
    const bool inx = gx >= 0 && gx < w, own = lane >= 2 && lane <= 29 && gx < w;
    auto load = [&](int y) { return row_ops(b, wd, ax, ay, dinv, inx && y >= 0 && y < h, (size_t)y * w + gx); };
    // rows t, t-1, t-2 of the operands and of x0; t-1, t-2, t-3 of x1
    RowOps q2{}, q1 = load(y0 - 2), q0 = load(y0 - 1), qn;
    float a2 = 0.f;                                                // x0 of row t-2
    float a1 = rbf(MG_OMEGA * q1.dinv * q1.b), s2 = 0.f, s3 = 0.f, o3ay = 0.f, o = 0.f;  // x0 of t-1; x1 of t-2 and t-3
    for (int t = y0 - 1; t < y1 + 2; t++) {
        // q0 is row t; its successor on the way
        qn = load(t + 1);
        const float a0 = rbf(MG_OMEGA * q0.dinv * q0.b);
        // x1 of row t-1
        const float al1 = from_left(q1.ax), xl = from_left(a1), xr = from_right(a1);
        float s1 = 0.f;
        {
            const int y = t - 1;
            if (inx && y >= 0 && y < h) s1 = rbf(a1 + MG_OMEGA * q1.dinv * resid_h(q1, al1, q2.ay, a1, xl, xr, a2, a0, gx, y, w, h));
        }
        // the residual of row t-2
        const int y = t - 2;
        const float al2 = from_left(q2.ax), sl = from_left(s2), sr = from_right(s2);
        float r = 0.f;
        const bool row = y >= y0 && y < y1;
        if (own && row) {
            sth(x, (size_t)y * w + gx, s2);
            r = rbf(resid_h(q2, al2, o3ay, s2, sl, sr, s3, s1, gx, y, w, h));
        }
        const float r1 = from_right(r);
        if (row) {
            if (!(y & 1)) o = 0.f;
            o += r;
            if (gx + 1 < w) o += r1;
            if (own && !(gx & 1) && ((y & 1) || y + 1 == h)) sth(cb, (size_t)(y >> 1) * cw + (gx >> 1), o);
        }
        o3ay = q2.ay;
        s3 = s2;
        s2 = s1;
        a2 = a1;
        a1 = a0;
        q2 = q1;
        q1 = q0;
        q0 = qn;
    }
}
// Up: x2 = x1 + P x_c, then two sweeps; the result -> out (BF16, or level 0's FP32 z with r.z: DOT, b is the CG's r).
template <class BT, class OT, bool DOT>
__global__ void __launch_bounds__(256) vc_up_h_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ xc, int cw,
                                                      const BT* __restrict__ b, const uint16_t* __restrict__ wd,
                                                      const uint16_t* __restrict__ ax, const uint16_t* __restrict__ ay,
                                                      const uint16_t* __restrict__ dinv, OT* __restrict__ out, int w, int h, const Strip S,
                                                      const CgRef C) {
    if (DOT && C.ctl[0]) return;
    const int lane = threadIdx.x & 31, wid = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int gx = wid % S.nx * 28 + lane - 2, y0 = wid / S.nx * S.rows, y1 = wid < S.warps ? min(h, y0 + S.rows) : 0;
    const bool inx = gx >= 0 && gx < w, own = lane >= 2 && lane <= 29 && gx < w;
    auto load = [&](int y) { return row_ops(b, wd, ax, ay, dinv, inx && y >= 0 && y < h, (size_t)y * w + gx); };
    auto X = [&](int y) { return inx && y >= 0 && y < h ? rbf(ldh(x, (size_t)y * w + gx) + ldh(xc, (size_t)(y >> 1) * cw + (gx >> 1))) : 0.f; };
    double v[1] = {0.0};
    if (y0 < y1) {
        RowOps q2{}, q1 = load(y0 - 2), q0 = load(y0 - 1), qn;
        float a2 = 0.f, a1 = X(y0 - 2), a0 = X(y0 - 1), s2 = 0.f, s3 = 0.f, o3ay = 0.f;
        for (int t = y0 - 1; t < y1 + 2; t++) {
            qn = load(t + 1);
            const float an = X(t + 1);
            // the first sweep of row t-1
            const float al1 = from_left(q1.ax), xl = from_left(a1), xr = from_right(a1);
            float s1 = 0.f;
            {
                const int y = t - 1;
                if (inx && y >= 0 && y < h) s1 = rbf(a1 + MG_OMEGA * q1.dinv * resid_h(q1, al1, q2.ay, a1, xl, xr, a2, a0, gx, y, w, h));
            }
            // the second of row t-2
            const int y = t - 2;
            const float al2 = from_left(q2.ax), sl = from_left(s2), sr = from_right(s2);
            if (own && y >= y0 && y < y1) {
                const float o = s2 + MG_OMEGA * q2.dinv * resid_h(q2, al2, o3ay, s2, sl, sr, s3, s1, gx, y, w, h);
                stv(out, (size_t)y * w + gx, o);
                if (DOT) v[0] += (double)q2.b * (double)o;
            }
            o3ay = q2.ay;
            s3 = s2;
            s2 = s1;
            a2 = a1;
            a1 = a0;
            a0 = an;
            q2 = q1;
            q1 = q0;
            q0 = qn;
        }
    }
    if (DOT && reduce_last(v, C.part, C.ctl + 2) && threadIdx.x == 0) cg_rz(C, v[0]);
}

// The coarsest level's sweeps in one cluster of 8 CTAs: each holds a band of rows, operators and both x buffers in
// shared memory, a warp per row; a sweep writes its band's first and last row into the neighbours' halo rows too
// (distributed shared memory) and ends in a cluster barrier. The zero-start sweep, then sweeps - 1 damped Jacobi ones,
// the result to x. What bounds it: the barrier and one pass over a few rows per warp (133 x 89 cells: 153 us in one
// CTA, 48 here); the bands hold levels of up to about 90 k cells, which fell to a launch per sweep before.
constexpr int CH_CTAS = 8, CH_THREADS = 512;
constexpr size_t CH_MAX_SMEM = 220 * 1024;
static size_t coarse_h_smem(const WlsLevel& L) {
    const size_t rows = (L.h + CH_CTAS - 1) / CH_CTAS;
    return sizeof(uint16_t) * L.w * (rows * 4 + (rows + 1) + 2 * (rows + 2));
}
static bool coarse_h_fits(const WlsLevel& L) { return coarse_h_smem(L) <= CH_MAX_SMEM; }
__global__ void __launch_bounds__(CH_THREADS) coarse_h_kernel(uint16_t* __restrict__ x, const uint16_t* __restrict__ b,
                                                              const uint16_t* __restrict__ wd, const uint16_t* __restrict__ ax,
                                                              const uint16_t* __restrict__ ay, const uint16_t* __restrict__ dinv, int w, int h,
                                                              int sweeps) {
    extern __shared__ uint16_t csm[];
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), rows = (h + CH_CTAS - 1) / CH_CTAS, r0 = rank * rows, nr = max(0, min(rows, h - r0));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint16_t *sb = csm, *swd = sb + rows * w, *sax = swd + rows * w, *sdi = sax + rows * w;
    uint16_t* say = sdi + rows * w;              // from the row above the band on
    uint16_t* xb[2] = {say + (rows + 1) * w, say + (rows + 1) * w + (rows + 2) * w};  // from the row above to the row below
    for (int k = tid; k < nr * w; k += CH_THREADS) {
        const size_t q = (size_t)r0 * w + k;
        sb[k] = b[q];
        swd[k] = wd[q];
        sax[k] = ax[q];
        sdi[k] = dinv[q];
        say[w + k] = ay[q];
    }
    if (r0 > 0 && nr > 0)
        for (int k = tid; k < w; k += CH_THREADS) say[k] = ay[(size_t)(r0 - 1) * w + k];
    uint16_t* up[2] = {nullptr, nullptr};    // the band above's lower halo row, the band below's upper one
    uint16_t* down[2] = {nullptr, nullptr};
    for (int q = 0; q < 2; q++) {
        if (rank > 0) up[q] = cl.map_shared_rank(xb[q], rank - 1) + (rows + 1) * w;  // every band above a band is whole
        if (rank + 1 < CH_CTAS) down[q] = cl.map_shared_rank(xb[q], rank + 1);
    }
    auto put = [&](int q, int r, int i, float v) {
        const bf e = __float2bfloat16_rn(v);
        const uint16_t u = *(const uint16_t*)&e;
        xb[q][(r + 1) * w + i] = u;
        if (r == 0 && up[q]) up[q][i] = u;
        if (r == nr - 1 && down[q]) down[q][i] = u;
    };
    cl.sync();  // this band is loaded, and every CTA runs: its neighbours may write into its halo rows
    for (int r = warp; r < nr; r += CH_THREADS / 32)
        for (int i = lane; i < w; i += 32) put(0, r, i, MG_OMEGA * ldh(sdi, r * w + i) * ldh(sb, r * w + i));
    cl.sync();
    for (int sw = 1; sw < sweeps; sw++) {
        const uint16_t* src = xb[(sw - 1) & 1];
        for (int r = warp; r < nr; r += CH_THREADS / 32) {
            const bool top = r0 + r > 0, bot = r0 + r + 1 < h;
            for (int i = lane; i < w; i += 32) {
                const int k = r * w + i, c = k + w;  // c: the cell in the x buffers and in say
                const float xk = ldh(src, c);
                float v = ldh(swd, k) * xk;
                if (i > 0) v += ldh(sax, k - 1) * (xk - ldh(src, c - 1));
                if (i + 1 < w) v += ldh(sax, k) * (xk - ldh(src, c + 1));
                if (top) v += ldh(say, c - w) * (xk - ldh(src, c - w));
                if (bot) v += ldh(say, c) * (xk - ldh(src, c + w));
                put(sw & 1, r, i, xk + MG_OMEGA * ldh(sdi, k) * (ldh(sb, k) - v));
            }
        }
        cl.sync();
    }
    const uint16_t* res = xb[(sweeps - 1) & 1] + w;
    for (int k = tid; k < nr * w; k += CH_THREADS) x[(size_t)r0 * w + k] = res[k];
}

WlsSolver* wls_alloc(int w, int h, cudaError_t* err) {
    *err = cudaSuccess;
    // set here, outside the graph captures of the CG iteration that launch it
    *err = cudaFuncSetAttribute(coarse_h_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CH_MAX_SMEM);
    if (*err == cudaSuccess) *err = cudaFuncSetAttribute(vcycle_tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_MAX_SMEM);
    if (*err != cudaSuccess) return nullptr;
    WlsSolver* S = new WlsSolver();
    S->w = w;
    S->h = h;
    const size_t n = (size_t)w * h;
    for (int cw = w, ch = h;; cw = (cw + 1) / 2, ch = (ch + 1) / 2) {
        WlsLevel L{};
        L.w = cw;
        L.h = ch;
        S->lv.push_back(L);
        if (std::max(cw, ch) <= MG_MIN) break;
    }
    // the planes laid out in one slab, 256-byte aligned: first their total, then their places
    for (int pass = 0; pass < 2; pass++) {
        size_t at = 0;
        auto put = [&](auto** p, size_t count) {
            using T = std::remove_pointer_t<std::remove_reference_t<decltype(*p)>>;
            if (pass) *p = (T*)((char*)S->slab + at);
            at += (count * sizeof(T) + 255) / 256 * 256;
        };
        for (WlsLevel& L : S->lv) {
            const size_t m = (size_t)L.w * L.h;
            for (float** q : {&L.wd, &L.ax, &L.ay, &L.dinv, &L.x, &L.b, &L.r}) put(q, m);
            for (uint16_t** q : {&L.hwd, &L.hax, &L.hay, &L.hdinv, &L.hx, &L.hb, &L.hr}) put(q, m);
        }
        for (float** q : {&S->ex, &S->ey, &S->cp, &S->dp, &S->f, &S->r, &S->z, &S->p, &S->p2, &S->ap}) put(q, n);
        put(&S->part, (size_t)2 * std::max(RED_BLOCKS, std::max(strip_blocks(strip_of(w, h, 1)), strip_blocks(strip_of(w, h, 2)))));
        put(&S->scal, 4);
        put(&S->alpha_beta, 4);
        put(&S->ctl, 4);
        if (pass == 0) {
            S->bytes = at;
            *err = lsb_dev_alloc(&S->slab, at);
            if (*err != cudaSuccess) return S;
        }
    }
    if (cudaHostAlloc((void**)&S->host_rel, 64, cudaHostAllocDefault) != cudaSuccess) *err = cudaErrorMemoryAllocation;
    for (cudaEvent_t& v : S->done)
        if (*err == cudaSuccess) *err = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
    return S;
}

cudaError_t wls_prepare(WlsSolver* S, const float* guide, float lambda, float sigma_c, int edge_mode, cudaStream_t) {
    S->lambda = lambda;
    S->inv = -1.0f / std::max(sigma_c, 1e-6f);
    S->inv2s2 = 1.0f / (2.0f * sigma_c * sigma_c);
    S->edge_mode = edge_mode;
    S->guide = guide;
    return cudaSuccess;
}

int wls_width(const WlsSolver* s) { return s->w; }
int wls_height(const WlsSolver* s) { return s->h; }
size_t wls_bytes(const WlsSolver* s) { return s ? s->bytes : 0; }

void wls_destroy(WlsSolver* s) {
    if (!s) return;
    if (s->g) cudaGraphExecDestroy(s->g);
    for (cudaEvent_t v : s->done)
        if (v) cudaEventDestroy(v);
    if (s->slab) cudaFree(s->slab);
    if (s->host_rel) cudaFreeHost(s->host_rel);
    delete s;
}

int wls_levels(const WlsSolver* s) { return (int)s->lv.size(); }

static bool tail_level(const WlsSolver* S, size_t l) {
    return (size_t)S->lv[l].w * S->lv[l].h <= (size_t)MG_TAIL_CELLS && S->lv.size() - l <= (size_t)MG_TAIL_MAX &&
           tail_floats(S, l) * sizeof(float) <= TAIL_MAX_SMEM;  // a long thin grid's levels only halve
}
static CgRef cg_ref(const WlsSolver* S) { return CgRef{S->part, S->scal, S->alpha_beta, S->ctl, (CgOut*)S->host_rel}; }

// Every level's operators: level 0 in one pass, each large level in one from the finer one, the small ones in one CTA;
// the edges too after a wls_prepare. mode 1: their BF16 copies on the levels its V-cycle visits. (As one kernel per
// quantity and level, with the copies made in both modes, this was 44 launches of a few us for a 1024 x 768 grid.)
cudaError_t wls_set_weights(WlsSolver* S, const float* conf, int mode, cudaStream_t s) {
    const float* guide = S->guide;
    S->guide = nullptr;
    auto ops = [&](size_t l) {
        const WlsLevel& C = S->lv[l];
        return mode == 1 && l < (size_t)MG_H_LEVELS ? HOps{C.hwd, C.hax, C.hay, C.hdinv} : HOps{};
    };
    const WlsLevel& Z = S->lv[0];
    auto level0 = [&](auto k) {
        lsb_launched(), k<<<g2(Z.w, Z.h), B2, 0, s>>>(guide, conf, Z.w, Z.h, S->inv, S->inv2s2, S->edge_mode, S->lambda, S->ex, S->ey, Z.ax, Z.ay,
                                                    Z.wd, Z.dinv, ops(0));
    };
    if (guide) level0(level0_kernel<true>);
    else level0(level0_kernel<false>);
    size_t l = 1;
    for (; l < S->lv.size() && !tail_level(S, l); l++) {
        const WlsLevel &F = S->lv[l - 1], &C = S->lv[l];
        if (guide) lsb_launched(), coarse_level_kernel<true><<<g2(C.w, C.h), B2, 0, s>>>(F, C, ops(l));
        else lsb_launched(), coarse_level_kernel<false><<<g2(C.w, C.h), B2, 0, s>>>(F, C, ops(l));
    }
    if (l < S->lv.size()) {
        MgSetup T;
        T.n = 0;
        for (size_t q = l - 1; q < S->lv.size(); q++, T.n++) T.lv[T.n] = S->lv[q], T.H[T.n] = ops(q);
        if (guide) lsb_launched(), coarse_tail_kernel<true><<<1, 1024, 0, s>>>(T);
        else lsb_launched(), coarse_tail_kernel<false><<<1, 1024, 0, s>>>(T);
    }
    return cudaGetLastError();
}

// depth.rs:924 `vcycle` (MG_PRE = MG_POST = 1): a level's way down and its way up in one pass each, the small levels in
// one CTA (every chain of levels ends in them: the coarsest has at most 16 x 16 cells). The right-hand side is bin
// (null: the level's b); the result lands in xout (null: the level's x, through its r buffer), with r.z at level 0.
static void vcycle(WlsSolver* S, size_t l, const float* bin, float* xout, cudaStream_t s) {
    WlsLevel& T = S->lv[l];
    if (tail_level(S, l)) {
        MgTail tl;
        tl.n = (int)(S->lv.size() - l);
        for (int q = 0; q < tl.n; q++) tl.lv[q] = S->lv[l + q];
        lsb_launched(), vcycle_tail_kernel<<<1, TAIL_THREADS, tail_floats(S, l) * sizeof(float), s>>>(tl);
        return;
    }
    WlsLevel& C = S->lv[l + 1];
    const float* b = bin ? bin : T.b;
    const Strip st = strip_of(T.w, T.h, 1);
    lsb_launched(), vc_down_kernel<<<strip_blocks(st), 256, 0, s>>>(b, T.wd, T.ax, T.ay, T.dinv, T.x, T.w, T.h, C.b, C.w, st);
    vcycle(S, l + 1, nullptr, nullptr, s);
    if (xout) {
        lsb_launched(), vc_up_kernel<true><<<strip_blocks(st), 256, 0, s>>>(T.x, C.x, C.w, b, T.wd, T.ax, T.ay, T.dinv, xout, T.w, T.h, st, cg_ref(S));
        return;
    }
    lsb_launched(), vc_up_kernel<false><<<strip_blocks(st), 256, 0, s>>>(T.x, C.x, C.w, b, T.wd, T.ax, T.ay, T.dinv, T.r, T.w, T.h, st, cg_ref(S));
    std::swap(T.x, T.r);
}

// A damped Jacobi sweep on level L (zero: the zero-start one) against its BF16 right-hand side:
// the coarsest level's sweeps when its bands do not fit the shared memory of coarse_h_kernel's cluster.
static void jacobi_h(WlsLevel& L, bool zero, cudaStream_t s) {
    if (zero) {
        lsb_launched(), jac0_h_kernel<uint16_t><<<g1((size_t)L.w * L.h), 256, 0, s>>>(L.hb, L.hdinv, L.hx, (size_t)L.w * L.h);
        return;
    }
    lsb_launched(), stencil_h_kernel<uint16_t, uint16_t><<<g2(L.w, L.h), B2, 0, s>>>(L.hx, L.hb, L.hwd, L.hax, L.hay, L.hdinv, L.hr, L.w,
                                                                                   L.h, 2);
    std::swap(L.hx, L.hr);
}
// the mixed-precision V-cycle: MG_H_SWEEPS pre/post sweeps, MG_H_LEVELS levels, MG_COARSE sweeps on
// the coarsest (one cluster). b32 / z32: level 0 takes the CG's FP32 residual as its right-hand side and
// its last sweep writes the FP32 z (no conversion passes).
static void vcycle_h(WlsSolver* S, size_t l, cudaStream_t s, const float* b32 = nullptr, float* z32 = nullptr) {
    WlsLevel& T = S->lv[l];
    const size_t last = std::min(S->lv.size(), (size_t)MG_H_LEVELS) - 1;
    if (l == last) {
        if (coarse_h_fits(T)) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(CH_CTAS);
            cfg.blockDim = dim3(CH_THREADS);
            cfg.dynamicSmemBytes = coarse_h_smem(T);  // wls_alloc raised the kernel's limit
            cfg.stream = s;
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = CH_CTAS;
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            lsb_launched();
            cudaLaunchKernelEx(&cfg, coarse_h_kernel, T.hx, (const uint16_t*)T.hb, (const uint16_t*)T.hwd, (const uint16_t*)T.hax,
                               (const uint16_t*)T.hay, (const uint16_t*)T.hdinv, T.w, T.h, MG_COARSE);
        } else {
            for (int k = 0; k < MG_COARSE; k++) jacobi_h(T, k == 0, s);
        }
        return;
    }
    static_assert(MG_H_SWEEPS == 2, "the fused BF16 passes run the zero-start sweep and one more down, two up");
    auto down_up = [&](auto* b) {  // the way down and the way up in one pass each
        using BT = std::remove_cv_t<std::remove_pointer_t<decltype(b)>>;
        WlsLevel& C = S->lv[l + 1];
        const Strip st = strip_of(T.w, T.h, 2);
        lsb_launched(), vc_down_h_kernel<BT><<<strip_blocks(st), 256, 0, s>>>(b, T.hwd, T.hax, T.hay, T.hdinv, T.hx, T.w, T.h, C.hb, C.w, st);
        vcycle_h(S, l + 1, s);
        if (z32) {
            lsb_launched(), vc_up_h_kernel<BT, float, true><<<strip_blocks(st), 256, 0, s>>>(T.hx, C.hx, C.w, b, T.hwd, T.hax, T.hay, T.hdinv, z32, T.w,
                                                                                          T.h, st, cg_ref(S));
        } else {
            lsb_launched(), vc_up_h_kernel<BT, uint16_t, false><<<strip_blocks(st), 256, 0, s>>>(T.hx, C.hx, C.w, b, T.hwd, T.hax, T.hay, T.hdinv,
                                                                                              T.hr, T.w, T.h, st, cg_ref(S));
            std::swap(T.hx, T.hr);
        }
    };
    if (b32) down_up(b32);
    else down_up((const uint16_t*)T.hb);
}

cudaError_t wls_solve(WlsSolver* S, const float* d, int max_iters, float* u, float* rel_out, int* iters_out, cudaStream_t s,
                      int mode, bool x0_given, double* rel64) {
    const int w = S->w, h = S->h;
    const size_t n = (size_t)w * h;
    WlsLevel& L0 = S->lv[0];
    if (w == 1 || h == 1) {
        // one line: the sweep is the answer, so it is the reference's, in its order (0.3 us a cell; a partition's error
        // against 64 bits is up to twice as large)
        lsb_launched();
        if (h == 1) thomas_kernel<true><<<1, TT, 0, s>>>(u, d, L0.wd, 0, S->ex, w, h, S->lambda, S->cp, S->dp);
        else thomas_kernel<false><<<1, TT, 0, s>>>(u, d, L0.wd, 0, S->ey, w, h, S->lambda, S->cp, S->dp);
        *rel_out = 0.f;
        *iters_out = 0;
        if (rel64) *rel64 = 0.0;
        return cudaGetLastError();
    }
    if (!x0_given) {
        // depth.rs:1022-1034: three separable sweeps, the first confidence-weighted
        const float* from = d;
        for (int t = 1; t <= 3; t++) {
            float p4 = 1.f;
            for (int q = 0; q < 3 - t; q++) p4 *= 4.f;
            const float lam_t = (1.5f * S->lambda * p4) / (64.f - 1.f);
            // rows into f, columns into u: no sweep reads what it writes
            cudaError_t e = thomas(true, S->f, from, L0.wd, t == 1 ? 0 : 1, S->ex, w, h, lam_t, S->cp, S->dp, S->z, s);
            if (e == cudaSuccess) e = thomas(false, u, S->f, L0.wd, 1, S->ey, w, h, lam_t, S->cp, S->dp, S->z, s);
            if (e != cudaSuccess) return e;
            from = u;
        }
    }
    const CgRef C = cg_ref(S);
    CgOut* host = (CgOut*)S->host_rel;
    const Strip st = strip_of(w, h, 1);
    // b = W d, |b|, r = b - A u; the reductions' ticket starts at 0, and every reduction leaves it there
    if (!S->ctl_zero) cudaMemsetAsync(S->ctl, 0, 4 * sizeof(int), s), S->ctl_zero = true;
    lsb_launched(), cg_start_kernel<<<strip_blocks(st), 256, 0, s>>>(d, u, L0.wd, L0.ax, L0.ay, S->r, w, h, st, C);
    const int nb1 = (int)std::min<size_t>(RED_BLOCKS, (n + 255) / 256);
    // z = M r and r.z
    auto precond = [&]() {
        if (mode == 1) {
            if (std::min(S->lv.size(), (size_t)MG_H_LEVELS) > 1) {  // r in, z out, no conversion passes
                vcycle_h(S, 0, s, S->r, S->z);
                return;
            }
            lsb_launched(), to_bf16_kernel<<<g1(n), 256, 0, s>>>(S->r, L0.hb, n);
            vcycle_h(S, 0, s);
            lsb_launched(), from_bf16_kernel<<<g1(n), 256, 0, s>>>(S->lv[0].hx, S->z, n);
        } else {
            if (!tail_level(S, 0)) {  // r in, z out: no copies
                vcycle(S, 0, S->r, S->z, s);
                return;
            }
            cudaMemcpyAsync(L0.b, S->r, n * sizeof(float), cudaMemcpyDeviceToDevice, s);
            vcycle(S, 0, nullptr, nullptr, s);
            cudaMemcpyAsync(S->z, S->lv[0].x, n * sizeof(float), cudaMemcpyDeviceToDevice, s);
        }
        lsb_launched(), cg_rz_kernel<<<nb1, 256, 0, s>>>(S->r, S->z, n, C);
    };
    auto iteration = [&]() {
        precond();
        lsb_launched(), cg_dir_kernel<<<strip_blocks(st), 256, 0, s>>>(S->z, S->p, S->p2, L0.wd, L0.ax, L0.ay, S->ap, w, h, st, C);
        lsb_launched(), cg_step_kernel<<<nb1, 256, 0, s>>>(u, S->p, S->p2, S->r, S->ap, n, max_iters, C);
    };
    // Every V-cycle restarts each level from zero, so which of a level's two buffers holds x
    // carries nothing from one cycle to the next: one captured iteration serves them all.
    bool graph = max_iters > 0;
    if (graph && (!S->g || S->g_u != u || S->g_mode != mode || S->g_max != max_iters)) {
        if (S->g) cudaGraphExecDestroy(S->g);
        S->g = nullptr;
        cudaGraph_t g = nullptr;
        const uint64_t c0 = lsb_launched_now();
        if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            iteration();
            const cudaError_t ec = cudaStreamEndCapture(s, &g);
            S->g_kernels = (long long)(lsb_launched_now() - c0);
            lsb_launched_add(-S->g_kernels);  // captured, not launched
            if (ec != cudaSuccess || !g || cudaGraphInstantiate(&S->g, g, 0) != cudaSuccess) S->g = nullptr;
            if (g) cudaGraphDestroy(g);
        }
        if (S->g) S->g_u = u, S->g_mode = mode, S->g_max = max_iters;
        else cudaGetLastError(), graph = false;  // launched directly instead
    }
    // Iterations are queued one ahead of the result the host has seen: the GPU does not wait for the host between
    // them (25 us each), and the one queued past the last does nothing (every kernel that changes the solution, the
    // residual or the result sees the stop word; the solution is the one a wait per iteration gives).
    cudaError_t e = cudaSuccess;
    for (int it = 0; it < max_iters; it++) {
        if (it >= 2) {
            e = cudaEventSynchronize(S->done[it & 1]);  // iteration it - 2
            if (e != cudaSuccess) return e;
            if (*(volatile int*)&host->stop) break;
        }
        if (graph) {
            e = cudaGraphLaunch(S->g, s);
            lsb_launched_add(S->g_kernels);
        } else {
            iteration();
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaEventRecord(S->done[it & 1], s);
        if (e != cudaSuccess) return e;
    }
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    *rel_out = host->rel;
    *iters_out = host->iters;
    if (rel64) *rel64 = host->rel64;
    return cudaGetLastError();
}

}  // namespace lsb
