// The fold: Burt-Adelson Laplacian pyramid + Wang-Chang region-energy
// selection over ALL frames of a stack.
//
// Reference semantics (crates/lapstack-core/src): per frame, pyramid.rs:203
// `build` (REDUCE pyramid.rs:86, EXPAND pyramid.rs:143, L = G - EXPAND),
// fuse.rs:200 `region_energy` (Y^2 of fuse.rs:160 through the binomial
// window of fuse.rs:168) and the strict-> winner-take-all of fuse.rs:414-451
// (ties to the earlier frame), frames folded in order.
//
// B200 layout: level-major instead of frame-major. Whoever owns a tile of level
// l walks the frames k = 0..n-1: L_l = G_l - EXPAND(G_{l+1}), the luma energy
// and its window sum, and the running best energy, winning coefficients and
// winner index stay on the SM. The accumulator is written once per level instead
// of read-modified-written once per frame. Level 0 of 16-bit frames is one kernel
// (lsb_fold0.cuh): REDUCE to G_1, the selection and the depth pass's focus slice
// (depth.rs:1097: luma -> ring difference filter -> block mean) from one staged
// copy of the interleaved u16 frame, its gains applied on load. The other levels
// are REDUCEd one after another (lsb_level.cuh), then selected together in one
// launch (lsb_select.cuh).
//
// Every float op on the selection path is an explicit round-to-nearest
// intrinsic in the reference's association order, so selection maps and
// coefficients are bit-identical to the reference FP32 CPU path.
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "lsb_common.cuh"
#include "lsb_internal.h"
#include "lsb_interp.cuh"

namespace lsb {

#include "lsb_level.cuh"
#include "lsb_fold0.cuh"
#include "lsb_select.cuh"


// The taps live in constant memory, one copy per device for every engine on it: they are written
// (stream-ordered on s) only when they change, and an engine that finds them already requested
// makes its stream wait for that write. Engines that run at the same time must ask for the same taps.
static std::mutex g_taps_mu;
static std::map<int, std::pair<std::vector<float>, cudaEvent_t>> g_taps;
cudaError_t set_focus_taps(const float* taps3, int ntaps, cudaStream_t s) {
    if (ntaps > 64) return cudaErrorInvalidValue;
    int dev = 0;
    cudaError_t de = cudaGetDevice(&dev);
    if (de != cudaSuccess) return de;
    std::lock_guard<std::mutex> lk(g_taps_mu);
    auto& cur = g_taps[dev];
    const std::vector<float> want(taps3, taps3 + 3 * ntaps);
    if (cur.second && cur.first == want) return cudaStreamWaitEvent(s, cur.second, 0);
    if (!cur.second) {
        de = cudaEventCreateWithFlags(&cur.second, cudaEventDisableTiming);
        if (de != cudaSuccess) {
            cur.second = nullptr;
            return de;
        }
    }
    int off[64];
    float wgt[64];
    for (int q = 0; q < ntaps; q++) {
        off[q] = (int)taps3[3 * q] * RGW + (int)taps3[3 * q + 1];
        wgt[q] = taps3[3 * q + 2];
    }
    cudaError_t e = cudaMemcpyToSymbolAsync(c_taps, taps3, sizeof(float) * 3 * ntaps, 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(c_tapo, off, sizeof(int) * ntaps, 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(c_tapw, wgt, sizeof(float) * ntaps, 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaEventRecord(cur.second, s);
    cur.first = e == cudaSuccess ? want : std::vector<float>();
    return e;
}

template <class K>
static cudaError_t with_smem(K k, size_t smem) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// The fused level-0 kernel applies: 16-bit frames, one call doing the REDUCE and the selection of the
// same frames, no halo control, no focus slice or the default one (ring difference filter r 1..3 on
// 2x2 blocks), and a frame with interior tiles.
static bool fold0_applies(const FoldArgs& a, int src, bool focus, int R) {
    if (src != SRC_U16 || a.level != 0 || a.halo_mode != 0 || !a.select || a.red_n <= 0) return false;
    if (a.red_k0 != a.sel_k0 || a.red_n != a.sel_k1 - a.sel_k0) return false;
    if (focus && !(a.rdf13 && a.bk == 2 && a.focus_kind == 0)) return false;
    return fold0_count(fold0_range(a.W, a.H, R)) > 0;
}

// The level-0 tiles the fused kernel leaves, as rectangles: the rows above and below its tiles, the columns beside them.
static void fold0_border_rects(int W, int H, const Fold0Range& rg, SelBatch& T) {
    const int ya = 32, yb = std::min(H, 32 * rg.iy1), xa = 64, xb = std::min(W, 64 * rg.ix1);
    const int r[4][4] = {{0, 0, W, std::min(ya, H)}, {0, ya, std::min(xa, W), yb}, {xb, ya, W, yb}, {0, yb, W, H}};
    T.n = 0;
    for (const auto& q : r)
        if (q[2] > q[0] && q[3] > q[1]) T.r[T.n++] = {0, q[0], q[1], q[2], q[3]};
}
// The selection of T's rectangles. Where a level's tiles are too few for the GPU's warps, 2, 3 or all 6 warps of a CTA
// take a share of the frames each of one tile (not with halo control, which adds the frames up in order).
template <int SRC, class GS, int R>
static cudaError_t launch_select(SelBatch& T, cudaStream_t s) {
    auto tiles = [](const SelBatch::Rect& r) { return (long)((r.x1 - r.x0 + SS_W - 1) / SS_W) * ((r.y1 - r.y0 + SS_H - 1) / SS_H); };
    constexpr long WANT = 148 * SS_CTAS * SS_WARPS;
    int ctas = 0, limit = 0;
    bool beside = false;
    for (int i = 0; i < T.n; i++) {
        auto& r = T.r[i];
        const FoldArgs& a = T.a[r.lv];
        long have = 0;
        for (int q = 0; q < T.n; q++)
            if (T.r[q].lv == r.lv) have += tiles(T.r[q]);
        r.groups = 1;
        if (a.halo_mode == 0)
            for (int g : {2, 3, 6})
                if (have * r.groups < WANT && g <= a.sel_k1 - a.sel_k0) r.groups = g;
        const uintptr_t src = SRC == SRC_U16 ? 1 : SRC == SRC_F32 ? (uintptr_t)a.src_f32 : (uintptr_t)a.src_g;
        r.vec = (a.W & 1) == 0 && src % (2 * (SRC == SRC_G ? sizeof(GS) : sizeof(float))) == 0;
        const int per = SS_H * SS_WARPS / r.groups;
        r.ntx = (r.x1 - r.x0 + SS_W - 1) / SS_W;
        r.cta0 = ctas;
        ctas += r.ntx * ((r.y1 - r.y0 + per - 1) / per);
        beside = beside || a.beside;
        limit = a.cta_limit;
    }
    T.ctas = ctas;
    const size_t smem = beside ? std::max(SS_SMEM, BESIDE_SMEM) : SS_SMEM;  // one CTA per SM beside the registration chain
    const bool turns = limit > 0 && limit < ctas;
    auto k = turns ? select_strip_kernel<SRC, GS, R, true> : select_strip_kernel<SRC, GS, R, false>;
    cudaError_t e = with_smem(k, smem);
    if (e != cudaSuccess) return e;
    lsb_launched(), k<<<turns ? limit : ctas, SS_WARPS * 32, smem, s>>>(T);
    return cudaGetLastError();
}
template <class GS>
static cudaError_t select_stored(SelBatch& T, int r, cudaStream_t s) {
    return r == 0 ? launch_select<SRC_G, GS, 0>(T, s) : r == 1 ? launch_select<SRC_G, GS, 1>(T, s) : r == 2 ? launch_select<SRC_G, GS, 2>(T, s) : cudaErrorInvalidValue;
}
// The selection alone of n levels above level 0, in one launch: the small ones take 20 us each by themselves, most of
// it the launch, cold instructions and one tile's latency.
cudaError_t fold_select(const FoldArgs* lv, int n, int storage, int radius, cudaStream_t s) {
    for (int i = 0; i < n;) {
        SelBatch T{};
        for (; i < n && T.n < SS_MAX; i++) {
            T.a[T.n] = lv[i];
            T.r[T.n] = {T.n, 0, 0, lv[i].W, lv[i].H};
            T.n++;
        }
        const cudaError_t e = storage == STORE_UNORM16 ? select_stored<unorm16>(T, radius, s)
                              : storage == STORE_F16   ? select_stored<__half>(T, radius, s) : select_stored<float>(T, radius, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// One level: REDUCE the frames asked for (and take their focus slices at level 0), then select.
// Level 0 of 16-bit frames: the fused kernel on the interior tiles, the two kernels on the others.
template <int SRC, class GS, int R, bool FOCUS, class SS>
static cudaError_t launch_level(const FoldArgs& a0, cudaStream_t s, int grid_limit) {
    cudaError_t e = cudaSuccess;
    FoldArgs a = a0;
    int rtiles = ((a.W1 + RW - 1) / RW) * ((a.H1 + RH - 1) / RH);
    SelBatch T{};
    T.n = 1;
    T.r[0] = {0, 0, 0, a.W, a.H};
    if (SRC == SRC_U16 && !a0.no_fused && fold0_applies(a0, SRC, FOCUS, R)) {
        auto kf = fold0_kernel<GS, R, FOCUS, SS>;
        const size_t fsm = a.beside ? std::max((size_t)f0::SMEM, BESIDE_SMEM) : (size_t)f0::SMEM;
        e = with_smem(kf, fsm);
        if (e != cudaSuccess) return e;
        const Fold0Range rg = fold0_range(a.W, a.H, R);
        const int nf = fold0_count(rg);
        lsb_launched(), kf<<<std::min(nf, std::max(grid_limit, 1)), f0::NT0, fsm, s>>>(a);
        if (a.after_fused) cudaEventRecord(a.after_fused, s);
        if (a.between) cudaEventRecord(a.between, s);
        a.between = nullptr;
        a.fused0 = 1;
        a.f0r = R;
        // the REDUCE's tiles are the level-0 tiles' G_1 blocks
        rtiles = fold0_border_count((a.W + 63) / 64, (a.H + 31) / 32, rg);
        if (rtiles <= 0) return cudaGetLastError();
        fold0_border_rects(a.W, a.H, rg, T);
    }
    if (a.red_n > 0) {
        if constexpr (SRC != SRC_U16 && !FOCUS) {
            const uintptr_t from = SRC == SRC_F32 ? (uintptr_t)a.src_f32 : (uintptr_t)a.src_g;
            const int vec = (a.W & 1) == 0 && from % (2 * (SRC == SRC_G ? sizeof(GS) : sizeof(float))) == 0;
            const int ntx = (a.W1 + RS_W - 1) / RS_W, nty = (a.H1 + RS_H * RS_WARPS - 1) / (RS_H * RS_WARPS);
            lsb_launched(), reduce_strip_kernel<SRC, GS><<<dim3(ntx * nty, a.red_n, 3), RS_WARPS * 32, 0, s>>>(a, ntx, vec);
        } else {
            auto kr = reduce_level_kernel<SRC, GS, FOCUS, SS>;
            const size_t rsm = (size_t)RED_FLOATS * sizeof(float);
            cudaError_t e = with_smem(kr, rsm);
            if (e != cudaSuccess) return e;
            lsb_launched(), kr<<<dim3(rtiles, a.red_n), NT, rsm, s>>>(a);
        }
    }
    if (a.between) cudaEventRecord(a.between, s);
    if (a.select) {
        T.a[0] = a;
        if ((e = launch_select<SRC, GS, R>(T, s)) != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

template <int SRC, class GS, int R>
static cudaError_t pick_focus(const FoldArgs& a, bool focus, cudaStream_t s, int gl) {
    if (!focus) return launch_level<SRC, GS, R, false, float>(a, s, gl);
    // 16-bit storage keeps the focus slices in FP16 (relative precision is what the peak search needs)
    if (sizeof(GS) == 2) return launch_level<SRC, GS, R, true, __half>(a, s, gl);
    return launch_level<SRC, GS, R, true, float>(a, s, gl);
}

template <int SRC, class GS>
static cudaError_t pick_r(const FoldArgs& a, int r, bool focus, cudaStream_t s, int gl) {
    switch (r) {
        case 0: return pick_focus<SRC, GS, 0>(a, focus, s, gl);
        case 1: return pick_focus<SRC, GS, 1>(a, focus, s, gl);
        case 2: return pick_focus<SRC, GS, 2>(a, focus, s, gl);
        default: return cudaErrorInvalidValue;
    }
}

template <class GS>
static cudaError_t pick_src(const FoldArgs& a, int src_kind, int r, bool focus, cudaStream_t s, int gl) {
    switch (src_kind) {
        case SRC_U16: return pick_r<SRC_U16, GS>(a, r, focus, s, gl);
        case SRC_F32: return pick_r<SRC_F32, GS>(a, r, focus, s, gl);
        default: return pick_r<SRC_G, GS>(a, r, false, s, gl);
    }
}

// wav.rs:146-161 the weighted average's accumulation over the frames as folded (level 0's source and
// gains): per pixel, frame by frame in order, w = the frame's weight plane taken bilinearly to the pixel
// (depth.rs:201 upsample_bilinear), acc += w * v per channel, wsum += w; then acc / wsum clamped to [0, 1].
template <int SRC>
__global__ void wav_accumulate_kernel(const FoldArgs a, const float* __restrict__ wts, int n, int dw, int dh, int k,
                                      float* __restrict__ out) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= a.W || y >= a.H) return;
    const float inv = __fdiv_rn(1.f, (float)k);
    int x0, x1, y0, y1;
    float tx, ty;
    bil_axis(x, inv, dw, x0, x1, tx);
    bil_axis(y, inv, dh, y0, y1, ty);
    const size_t m = (size_t)dw * dh, np = (size_t)a.W * a.H, o = (size_t)y * a.W + x;
    float acc[3] = {0.f, 0.f, 0.f}, ws = 0.f;
    for (int f = 0; f < n; f++) {
        const float wv = bil(wts + (size_t)f * m, dw, x0, x1, y0, y1, tx, ty);
        float v[3];
        level_px<SRC, float>(a, f, x, y, v);
#pragma unroll
        for (int c = 0; c < 3; c++) acc[c] = __fadd_rn(acc[c], __fmul_rn(wv, v[c]));
        ws = __fadd_rn(ws, wv);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) out[c * np + o] = fminf(fmaxf(__fdiv_rn(acc[c], ws), 0.f), 1.f);
}

cudaError_t wav_accumulate(const FoldArgs& a, int src_kind, const float* wts, int n, int dw, int dh, int k, float* out, cudaStream_t s) {
    dim3 b(32, 8), g((a.W + 31) / 32, (a.H + 7) / 8);
    if (src_kind == SRC_F32) lsb_launched(), wav_accumulate_kernel<SRC_F32><<<g, b, 0, s>>>(a, wts, n, dw, dh, k, out);
    else if (src_kind == SRC_U16) lsb_launched(), wav_accumulate_kernel<SRC_U16><<<g, b, 0, s>>>(a, wts, n, dw, dh, k, out);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t fold_level(const FoldArgs& a0, int src_kind, int storage, int radius, bool focus, cudaStream_t s, int grid_limit) {
    const FoldArgs& a = a0;
    if (a.W <= 0 || a.H <= 0) return cudaSuccess;
    switch (storage) {
        case STORE_UNORM16: return pick_src<unorm16>(a, src_kind, radius, focus, s, grid_limit);
        case STORE_F16: return pick_src<__half>(a, src_kind, radius, focus, s, grid_limit);
        default: return pick_src<float>(a, src_kind, radius, focus, s, grid_limit);
    }
}

cudaError_t warp_frames(const uint16_t* frames, const FrameXform* xf, int interp, int w, int h, int n, bool u16_out, void* out,
                        cudaStream_t s) {
    if (interp == 3) {  // Spline4x4: the tiled form
        dim3 g((w + WT_W - 1) / WT_W, (h + WT_H - 1) / WT_H, n);
        if (u16_out) lsb_launched(), warp_tile_kernel<true><<<g, NT, 0, s>>>(frames, xf, w, h, out);
        else lsb_launched(), warp_tile_kernel<false><<<g, NT, 0, s>>>(frames, xf, w, h, out);
        return cudaGetLastError();
    }
    dim3 g((w + 31) / 32, (h + 7) / 8, n);
    if (u16_out) lsb_launched(), warp_frames_kernel<true><<<g, NT, 0, s>>>(frames, xf, interp, w, h, out);
    else lsb_launched(), warp_frames_kernel<false><<<g, NT, 0, s>>>(frames, xf, interp, w, h, out);
    return cudaGetLastError();
}

// ------------------------------------------------------------ residual level
// fuse.rs:207 `deviation_entropy` of each frame's top luma, one thread per
// (frame, pixel). lnp[c] = ln(c / n) as the reference's f32 ln gives it
// (computed on the host with the platform libm).
template <class GS>
__global__ void dev_ent_kernel(const ResidualArgs a, const float* __restrict__ lnp) {
    const int n2 = a.w * a.h;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= a.n * n2) return;
    const int k = idx / n2, pix = idx % n2, i = pix / a.w, j = pix % a.w;
    const GS* t = (const GS*)a.tops + (size_t)k * 3 * n2;
    const int r = a.radius, nwin = (2 * r + 1) * (2 * r + 1);
    const float inv_n = __fdiv_rn(1.f, (float)nwin);
    const float qscale = (float)(min(max(a.bins, 2), 65536) - 1);
    float s = 0.f, s2 = 0.f;
    int q[81];
    int m = 0;
    for (int dy = -r; dy <= r; dy++) {
        const int yy = lsb_reflect(i + dy, a.h);
        for (int dx = -r; dx <= r; dx++) {
            const int o = yy * a.w + lsb_reflect(j + dx, a.w);
            const float2 sc = make_float2(0.f, a.xf[k].ginv);
            const float v = lsb_luma(Store<GS>::ld(t + o, sc), Store<GS>::ld(t + n2 + o, sc), Store<GS>::ld(t + 2 * n2 + o, sc));
            s = __fadd_rn(s, v);
            s2 = __fadd_rn(s2, __fmul_rn(v, v));
            const float vc = fminf(fmaxf(v, 0.f), 1.f);
            q[m++] = (int)__fadd_rn(__fmul_rn(vc, qscale), 0.5f);
        }
    }
    const float mean = __fmul_rn(s, inv_n);
    a.dev[idx] = fmaxf(__fsub_rn(__fmul_rn(s2, inv_n), __fmul_rn(mean, mean)), 0.f);
    // entropy over the bins in order of first touch
    float e = 0.f;
    for (int u = 0; u < m; u++) {
        bool seen = false;
        for (int v = 0; v < u; v++) seen |= q[v] == q[u];
        if (seen) continue;
        int cnt = 0;
        for (int v = u; v < m; v++) cnt += q[v] == q[u];
        const float p = __fmul_rn((float)cnt, inv_n);
        e = __fsub_rn(e, __fmul_rn(p, lnp[cnt]));
    }
    a.ent[idx] = e;
}

// fuse.rs:248 the Pareto mean (or the plain mean) over the frames per pixel.
template <class GS>
__global__ void pareto_kernel(const ResidualArgs a) {
    const int n2 = a.w * a.h;
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= n2) return;
    float o[3] = {0.f, 0.f, 0.f};
    const GS* t = (const GS*)a.tops;
    if (a.n == 1 || a.top_rule == 2) {
        const float inv = __fdiv_rn(1.f, (float)a.n);
        for (int k = 0; k < a.n; k++) {
            const float2 sc = make_float2(0.f, a.xf[k].ginv);
            for (int c = 0; c < 3; c++) o[c] = __fadd_rn(o[c], __fmul_rn(Store<GS>::ld(t + ((size_t)k * 3 + c) * n2 + pix, sc), inv));
        }
    } else {
        const bool ent = a.top_rule == 0;
        auto dominated = [&](int x) {
            const float da = a.dev[(size_t)x * n2 + pix], ea = a.ent[(size_t)x * n2 + pix];
            for (int b = 0; b < a.n; b++) {
                if (b == x) continue;
                const float db = a.dev[(size_t)b * n2 + pix], eb = a.ent[(size_t)b * n2 + pix];
                const bool d = ent ? (db >= da && eb >= ea && (db > da || eb > ea)) : (db > da || (db == da && b < x));
                if (d) return true;
            }
            return false;
        };
        int kept = 0;
        for (int x = 0; x < a.n; x++) kept += !dominated(x);
        const float inv = __fdiv_rn(1.f, (float)max(kept, 1));
        for (int x = 0; x < a.n; x++)
            if (!dominated(x)) {
                const float2 sc = make_float2(0.f, a.xf[x].ginv);
                for (int c = 0; c < 3; c++) o[c] = __fadd_rn(o[c], __fmul_rn(Store<GS>::ld(t + ((size_t)x * 3 + c) * n2 + pix, sc), inv));
            }
    }
    for (int c = 0; c < 3; c++) a.out[(size_t)c * n2 + pix] = o[c];
}

template <class GS>
static void residual_launch(const ResidualArgs& a, const float* lnp, cudaStream_t s) {
    const int n2 = a.w * a.h;
    if (a.n > 1 && a.top_rule != 2) lsb_launched(), dev_ent_kernel<GS><<<(a.n * n2 + 127) / 128, 128, 0, s>>>(a, lnp);
    lsb_launched(), pareto_kernel<GS><<<(n2 + 127) / 128, 128, 0, s>>>(a);
}
cudaError_t fuse_residuals(const ResidualArgs& a, int storage, const float* lnp, cudaStream_t s) {
    if (a.radius > 4) return cudaErrorInvalidValue;
    if (storage == STORE_UNORM16) residual_launch<unorm16>(a, lnp, s);
    else if (storage == STORE_F16) residual_launch<__half>(a, lnp, s);
    else residual_launch<float>(a, lnp, s);
    return cudaGetLastError();
}

// ------------------------------------------------------------- halo control
// pyramid.rs:86 REDUCE of one f32 plane per frame: the 5 reflected rows each
// reduced along x (the row pass), then those 5 values along y (the column
// pass) -- the same operations, in the same order, as the two passes.
__global__ void reduce_weights_kernel(const float* __restrict__ src, int w, int h, float* __restrict__ dst, int w1, int h1) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    if (j >= w1 || i >= h1) return;
    const float* p = src + (size_t)k * w * h;
    float r[5];
    for (int t = 0; t < 5; t++) {
        const float* row = p + (size_t)lsb_reflect(2 * i + t - 2, h) * w;
        r[t] = lsb_tap5(row[lsb_reflect(2 * j - 2, w)], row[lsb_reflect(2 * j - 1, w)], row[lsb_reflect(2 * j, w)],
                        row[lsb_reflect(2 * j + 1, w)], row[lsb_reflect(2 * j + 2, w)]);
    }
    dst[(size_t)k * w1 * h1 + (size_t)i * w1 + j] = lsb_tap5(r[0], r[1], r[2], r[3], r[4]);
}
cudaError_t reduce_weights(const float* src, int w, int h, int n, float* dst, int w1, int h1, cudaStream_t s) {
    dim3 b(32, 8), g((w1 + 31) / 32, (h1 + 7) / 8, n);
    lsb_launched(), reduce_weights_kernel<<<g, b, 0, s>>>(src, w, h, dst, w1, h1);
    return cudaGetLastError();
}
// fuse.rs:466-470 at the top level: acc = G * w for frame 0, then acc += w * G; best = sum w
template <class GS>
__global__ void halo_top_kernel(const GS* __restrict__ tops, const FrameXform* __restrict__ xf, const float* __restrict__ wts, int n, int w,
                                int h, float* __restrict__ acc, float* __restrict__ best) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const size_t n2 = (size_t)w * h, o = (size_t)y * w + x;
    float a[3] = {0.f, 0.f, 0.f}, b = 0.f;
    for (int k = 0; k < n; k++) {
        const float2 sc = make_float2(xf[k].gscale, xf[k].ginv);
        const float wv = wts[(size_t)k * n2 + o];
        for (int c = 0; c < 3; c++) {
            const float g = Store<GS>::ld(tops + ((size_t)k * 3 + c) * n2 + o, sc);
            a[c] = k == 0 ? __fmul_rn(g, wv) : __fadd_rn(a[c], __fmul_rn(wv, g));
        }
        b = k == 0 ? wv : __fadd_rn(b, wv);
    }
    for (int c = 0; c < 3; c++) acc[c * n2 + o] = a[c];
    best[o] = b;
}
cudaError_t halo_top(const void* tops, int storage, const FrameXform* xf, const float* wts, int n, int w, int h, float* acc, float* best,
                     cudaStream_t s) {
    dim3 b(32, 8), g((w + 31) / 32, (h + 7) / 8);
    if (storage == STORE_UNORM16) lsb_launched(), halo_top_kernel<unorm16><<<g, b, 0, s>>>((const unorm16*)tops, xf, wts, n, w, h, acc, best);
    else if (storage == STORE_F16) lsb_launched(), halo_top_kernel<__half><<<g, b, 0, s>>>((const __half*)tops, xf, wts, n, w, h, acc, best);
    else lsb_launched(), halo_top_kernel<float><<<g, b, 0, s>>>((const float*)tops, xf, wts, n, w, h, acc, best);
    return cudaGetLastError();
}
// fuse.rs:508: the weighted means
__global__ void halo_divide_kernel(float* __restrict__ acc, const float* __restrict__ best, size_t n2) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n2; i += (size_t)gridDim.x * blockDim.x)
        for (int c = 0; c < 3; c++) acc[c * n2 + i] = __fdiv_rn(acc[c * n2 + i], best[i]);
}
cudaError_t halo_divide(float* acc, const float* best, int w, int h, cudaStream_t s) {
    const size_t n2 = (size_t)w * h;
    lsb_launched(), halo_divide_kernel<<<(int)std::min<size_t>((n2 + 255) / 256, 148 * 8), 256, 0, s>>>(acc, best, n2);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ collapse
// pyramid.rs:219: G_l = L_l + EXPAND(G_{l+1}), EXPAND horizontal then
// vertical (pyramid.rs:143) evaluated per output pixel with the same taps;
// at level 0 also fuse.rs:516 clamp and io.rs:287 u16 packing.
// In register strips: a warp takes 60 x `rows` pixels, a lane the coarse column under its pixel pair; the row taps'
// neighbours are shuffles, three expanded coarse rows stay in registers. What bounds it: its 33 bytes a pixel. One
// pixel a thread, with its 9 coarse values of each channel read again, took 0.79 ms at 6000 x 4000 (0.12 of reads and
// writes), 0.23 here; the five levels of 1024 x 768 68 us -> 27.
constexpr int CS_W = 60, CS_WARPS = 4;
template <bool LAST>
__global__ void __launch_bounds__(CS_WARPS * 32) collapse_kernel(const float* __restrict__ acc, const float* __restrict__ coarse,
                                                                 float* __restrict__ out, int w, int h, int cw, int ch, int ntx, int rows,
                                                                 uint16_t* __restrict__ rgb) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int cx = (int)(blockIdx.x % ntx) * (CS_W / 2) - 1 + lane, x = 2 * cx;
    const int y0 = ((int)(blockIdx.x / ntx) * CS_WARPS + wid) * rows;
    if (y0 >= h) return;
    const size_t np = (size_t)w * h, cp = (size_t)cw * ch;
    const bool own0 = lane >= 1 && lane <= CS_W / 2 && x < w, own1 = own0 && x + 1 < w;
    const bool vec = (w & 1) == 0;  // every row of pairs is aligned (the planes are the pool's own)
    const float* cc = coarse + lsb_reflect(cx, cw);
    auto load = [&](int cy, float v[3]) {
        const float* p = cc + (size_t)lsb_reflect(cy, ch) * cw;
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = p[c * cp];
    };
    auto expand = [&](const float v[3], float2 e[3]) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const float l = __shfl_up_sync(ALL, v[c], 1), r = __shfl_down_sync(ALL, v[c], 1);
            e[c] = make_float2(lsb_exp_even(l, v[c], r), lsb_exp_odd(v[c], r));
        }
    };
    float2 A[3], B[3], C[3];
    float n[3];
    {
        float v0[3], v1[3];
        load((y0 >> 1) - 1, v0);
        load(y0 >> 1, v1);
        load((y0 >> 1) + 1, n);
        expand(v0, B);
        expand(v1, C);
    }
#pragma unroll 2
    for (int y = y0; y < y0 + rows && y < h; y += 2) {
#pragma unroll
        for (int c = 0; c < 3; c++) A[c] = B[c], B[c] = C[c];
        expand(n, C);
        load((y >> 1) + 2, n);
#pragma unroll
        for (int s = 0; s < 2; s++) {
            if (y + s >= h) break;
            const size_t o = (size_t)(y + s) * w + x;
            float2 r[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float* p = acc + c * np + o;
                const float2 v = !own0 ? splat(0.f) : vec ? *(const float2*)p : make_float2(p[0], own1 ? p[1] : 0.f);
                r[c] = add2(v, s ? exp_odd2(B[c], C[c]) : exp_even2(A[c], B[c], C[c]));
                if (LAST) r[c] = make_float2(fminf(fmaxf(r[c].x, 0.f), 1.f), fminf(fmaxf(r[c].y, 0.f), 1.f));
                float* q = out + c * np + o;
                if (vec) {
                    if (own0) *(float2*)q = r[c];
                } else {
                    if (own0) q[0] = r[c].x;
                    if (own1) q[1] = r[c].y;
                }
            }
            if (LAST && rgb) {
                unsigned u[6];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    u[c] = (uint16_t)__fadd_rn(__fmul_rn(r[c].x, 65535.f), 0.5f);
                    u[3 + c] = (uint16_t)__fadd_rn(__fmul_rn(r[c].y, 65535.f), 0.5f);
                }
                uint16_t* q = rgb + o * 3;
                if (vec) {
                    unsigned* q4 = (unsigned*)q;
                    if (own0) q4[0] = u[0] | u[1] << 16, q4[1] = u[2] | u[3] << 16, q4[2] = u[4] | u[5] << 16;
                } else {
                    if (own0) q[0] = (uint16_t)u[0], q[1] = (uint16_t)u[1], q[2] = (uint16_t)u[2];
                    if (own1) q[3] = (uint16_t)u[3], q[4] = (uint16_t)u[4], q[5] = (uint16_t)u[5];
                }
            }
        }
    }
}

// fuse.rs:336 `upsample_index`: the depth level's winner map, nearest, to full size (clamped at the edge)
__global__ void upsample_index_kernel(const uint16_t* __restrict__ win, int dwl, int dhl, int scale, int w, int h, float* __restrict__ out) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    out[(size_t)y * w + x] = (float)win[(size_t)min(y / scale, dhl - 1) * dwl + min(x / scale, dwl - 1)];
}
cudaError_t upsample_index(const uint16_t* win, int dwl, int dhl, int scale, int w, int h, float* out, cudaStream_t s) {
    dim3 b(32, 8), g((w + 31) / 32, (h + 7) / 8);
    lsb_launched(), upsample_index_kernel<<<g, b, 0, s>>>(win, dwl, dhl, scale, w, h, out);
    return cudaGetLastError();
}

cudaError_t collapse_level(const float* acc, const float* coarse, float* out, int w, int h, int cw, int ch, bool last,
                           uint16_t* rgb_out, cudaStream_t s) {
    // 16 rows a warp, fewer while the level has too few of them to fill the GPU: a row pair takes a round of latency
    const int ntx = (w + CS_W - 1) / CS_W;
    int rows = 16;
    while (rows > 2 && (long)ntx * ((h + rows - 1) / rows) < 148 * 16) rows /= 2;
    const int g = ntx * ((h + rows * CS_WARPS - 1) / (rows * CS_WARPS));
    if (last) lsb_launched(), collapse_kernel<true><<<g, CS_WARPS * 32, 0, s>>>(acc, coarse, out, w, h, cw, ch, ntx, rows, rgb_out);
    else lsb_launched(), collapse_kernel<false><<<g, CS_WARPS * 32, 0, s>>>(acc, coarse, out, w, h, cw, ch, ntx, rows, rgb_out);
    return cudaGetLastError();
}

// ------------------------------------------------------------ winner shares
// fuse.rs:315 `winner_shares`: the plane's largest winning energy, then per frame the cells it
// wins above 1% of that.
__global__ void max_kernel(const float* __restrict__ v, int n, float* out) {
    float m = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = fmaxf(m, v[i]);
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax((int*)out, __float_as_int(m));  // non-negative floats order as ints
}
// What bounds it: atomic additions to few addresses (neighbours share a winner), one per cell in global memory: 2.8 M
// cells 1.78 ms. So a warp adds once per different winner among its 32 cells, into the CTA's table for the first
// COUNT_SH frames (the rest go to global memory directly), and a CTA adds its table once: 15 us.
constexpr int COUNT_SH = 1024;
__global__ void __launch_bounds__(256) count_kernel(const uint16_t* __restrict__ win, const float* __restrict__ best, int n, int frames,
                                                    const float* mx, unsigned int* counts) {
    __shared__ unsigned tab[COUNT_SH];
    for (int k = threadIdx.x; k < COUNT_SH; k += 256) tab[k] = 0;
    __syncthreads();
    const float fl = __fmul_rn(0.01f, *mx);
    const int lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * 256 + (threadIdx.x - lane); i0 < n; i0 += gridDim.x * 256) {
        const int i = i0 + lane;
        const int k = i < n && best[i] > fl && fl > 0.f && win[i] < frames ? win[i] : -1;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        if (k >= 0 && lane == __ffs(same) - 1) atomicAdd(k < COUNT_SH ? &tab[k] : &counts[k], (unsigned)__popc(same));
    }
    __syncthreads();
    for (int k = threadIdx.x; k < min(frames, COUNT_SH); k += 256)
        if (tab[k]) atomicAdd(&counts[k], tab[k]);
}
cudaError_t winner_counts(const uint16_t* win, const float* best, int cells, int frames, unsigned int* counts, float* mx,
                          cudaStream_t s) {
    cudaMemsetAsync(mx, 0, sizeof(float), s);
    cudaMemsetAsync(counts, 0, sizeof(unsigned int) * frames, s);
    int g = std::min((cells + 255) / 256, 148 * 4);
    lsb_launched(), max_kernel<<<g, 256, 0, s>>>(best, cells, mx);
    lsb_launched(), count_kernel<<<g, 256, 0, s>>>(win, best, cells, frames, mx, counts);
    return cudaGetLastError();
}

// ------------------------------------------------------- brightness means
// brightness.rs:67 `sums` at the identity over the stride-4 grid: per frame,
// per-block f64 partial sums (a fixed tree), then the partials in order.
__global__ void means_partial_kernel(const uint16_t* __restrict__ frames, int w, int h, int nparts, double* partial) {
    const int k = blockIdx.y, part = blockIdx.x;
    const int gw = (w + 3) / 4, gh = (h + 3) / 4, ng = gw * gh;
    const int per = (ng + nparts - 1) / nparts, lo = part * per, hi = min(ng, lo + per);
    const uint16_t* f = frames + (size_t)k * w * h * 3;
    double s[3] = {0.0, 0.0, 0.0};
    for (int g = lo + threadIdx.x; g < hi; g += blockDim.x) {
        const size_t i = (size_t)(g / gw) * 4 * w + (g % gw) * 4;
        for (int c = 0; c < 3; c++) s[c] += (double)__fmul_rn((float)f[i * 3 + c], LSB_INV16);
    }
    __shared__ double red[3][256];
    for (int c = 0; c < 3; c++) red[c][threadIdx.x] = s[c];
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st)
            for (int c = 0; c < 3; c++) red[c][threadIdx.x] += red[c][threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 3; c++) partial[((size_t)k * nparts + part) * 3 + c] = red[c][0];
}
// brightness.rs:67: each frame's partials summed in part order.
__global__ void means_final_kernel(const double* partial, int n, int nparts, int count, double* means) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    for (int c = 0; c < 3; c++) {
        double s = 0.0;
        for (int p = 0; p < nparts; p++) s += partial[((size_t)k * nparts + p) * 3 + c];
        means[k * 3 + c] = count == 0 ? 0.0 : s / (double)count;
    }
}
cudaError_t frame_means(const uint16_t* frames, int n, int w, int h, double* partial, int nparts, double* means, cudaStream_t s) {
    dim3 g(nparts, n);
    lsb_launched(), means_partial_kernel<<<g, 256, 0, s>>>(frames, w, h, nparts, partial);
    const int count = ((w + 3) / 4) * ((h + 3) / 4);
    lsb_launched(), means_final_kernel<<<(n + 127) / 128, 128, 0, s>>>(partial, n, nparts, count, means);
    return cudaGetLastError();
}

}  // namespace lsb
