// The selection of a pyramid level in register strips -- included by lsb_fold.cu inside namespace lsb, after
// lsb_fold0.cuh (whose packed f32x2 helpers it uses).
//
// A warp owns a tile of 56 x 8 pixels of level l and walks the frames in order; for each frame it forms
// L = G - EXPAND(G_{l+1}) (pyramid.rs:143/209), the node energy and its binomial window (fuse.rs:152/168) and keeps
// the strict-> selection (fuse.rs:429) of its pixels in shared memory, its own lanes' words, which are written only
// when a frame wins. Lane i holds the pixel pair (x0 - 4 + 2i, +1) and the G_{l+1} column under it, so EXPAND along
// rows and the window's columns are shuffles; lanes 2 .. 29 own pixels, the others are the window's reach. Rows run
// down the tile in pairs: three expanded G_{l+1} rows, 2R + 1 window row sums and R + 1 rows of L are live at a time,
// and the next pair's rows, or the next frame's first, are on their way.
// What bounds it: the latency of its loads, then instructions issued (300 per row pair of a warp, 75 a pixel). The
// kernel before it staged G_l and G_{l+1} of a 64 x 32 tile in shared memory, with a barrier between its passes.
// 3000 x 2000 f32, 8 frames, R = 1: 1.50 ms -> 0.26 (its reads and writes take 0.12); the five levels of a 1024 x 768
// stack of 8, now one launch: 0.24 ms -> 0.03.
// 6 warps a CTA and 3 CTAs an SM: with 4 (80 registers) it spills, 0.45 ms against 0.38 before the next frame's rows
// were loaded early; with the state in registers and the rows unrolled (168 registers) 0.55, and the coarse levels
// waited for instructions.
// Every float op is the reference's, in its order.
#pragma once

constexpr int SS_W = 56, SS_H = 8, SS_WARPS = 6, SS_CTAS = 3;

// What a launch selects: rectangles of tiles of one or more levels, one after another in the grid.
constexpr int SS_MAX = 16;
struct SelBatch {
    int n, ctas;  // rectangles; CTAs of work, which the launched ones take in turn
    struct Rect {
        int lv;                        // its level's arguments
        int x0, y0, x1, y1, ntx, cta0;  // cta0: the first CTA's index
        int vec;                       // rows of G_l are aligned pairs
        int groups;                    // 1, 2, 3 or 6: this many warps of a CTA split a tile's frames, merged in order (strict >)
    } r[SS_MAX];
    FoldArgs a[SS_MAX];
};

// A row of three channels at a lane's two columns.
template <int SRC, class GS, bool VEC>
__device__ __forceinline__ void ss_row(const FoldArgs& a, const void* f, size_t np, int off, int o1, float2 sc, float2 v[3]) {
    if (SRC == SRC_U16) {
        const uint16_t* p = (const uint16_t*)f + 3 * (size_t)off;
        const uint16_t* q = p + 3 * o1;
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = make_float2(__fmul_rn((float)p[c], LSB_INV16), __fmul_rn((float)q[c], LSB_INV16));
    } else if (SRC == SRC_F32) {
        const float* p = (const float*)f + off;
#pragma unroll
        for (int c = 0; c < 3; c++, p += np) v[c] = VEC ? *(const float2*)p : make_float2(p[0], p[o1]);
    } else if (VEC && sizeof(GS) == 2) {
        const GS* p = (const GS*)f + off;
#pragma unroll
        for (int c = 0; c < 3; c++, p += np) {
            const unsigned u = *(const unsigned*)p;
            GS e[2];
            *(uint16_t*)&e[0] = (uint16_t)u;
            *(uint16_t*)&e[1] = (uint16_t)(u >> 16);
            v[c] = make_float2(Store<GS>::ld(&e[0], sc), Store<GS>::ld(&e[1], sc));
        }
    } else if (VEC) {
        const float* p = (const float*)f + off;
#pragma unroll
        for (int c = 0; c < 3; c++, p += np) v[c] = *(const float2*)p;
    } else {
        const GS* p = (const GS*)f + off;
#pragma unroll
        for (int c = 0; c < 3; c++, p += np) v[c] = make_float2(Store<GS>::ld(p, sc), Store<GS>::ld(p + o1, sc));
    }
}

// A tile's state, 8 rows x 2 pixels a lane, in shared memory (it is written only when a frame wins):
// st[(9 j + w) * 32], w = 2 c + l the coefficients, 6 + l the energies, 8 the frames (16 bits each).
// Frames k0 .. k1 - 1 over a tile at (x0, y0), each one's first rows loaded while the one before ends. MODE 0: nothing of it meets the level's border, rows of 8-byte (4-byte) aligned
// pairs; 1: the same without the alignment; 2: any tile, and chroma and halo control.
template <int SRC, class GS, int R, int MODE>
__device__ __forceinline__ void ss_frames(const FoldArgs& a, int k0, int k1, int x0, int y0, int lane, float* st) {
    constexpr bool EDGE = MODE == 2;
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int NP = SS_H / 2 + R;  // row pairs: y0 - R + 2p, + 1
    constexpr bool ODD = R & 1;       // the pair's first row is odd
    const int W = a.W, H = a.H, W1 = a.W1, H1 = a.H1;
    const size_t np = (size_t)W * H, np1 = (size_t)W1 * H1;
    if (k0 >= k1) return;
    const int xb = x0 - 4, xl = xb + 2 * lane;
    // columns and rows beyond the level: the reflected ones (pyramid.rs:51), as EXPAND reads G_{l+1}
    const int xi0 = EDGE ? lsb_reflect(xl, W) : xl, xi1 = EDGE ? lsb_reflect(xl + 1, W) : xl + 1, o1 = xi1 - xi0;
    const int xg = EDGE ? lsb_reflect((x0 >> 1) - 2 + lane, W1) : (x0 >> 1) - 2 + lane;
    float2 sc, scn = make_float2(a.xf[k0].gscale, a.xf[k0].ginv);  // this frame's storage scale and the next one's
    float gain[3] = {1.f, 1.f, 1.f};
    auto load_g1 = [&](int k, float2 scale, int cy, float v[3]) {
        const GS* p = (const GS*)a.dst_g + (size_t)k * np1 * 3 + (size_t)(EDGE ? lsb_reflect(cy, H1) : cy) * W1 + xg;
#pragma unroll
        for (int c = 0; c < 3; c++, p += np1) v[c] = Store<GS>::ld(p, scale);
    };
    auto load_row = [&](int k, float2 scale, int y, float2 v[3]) {
        const void* f = SRC == SRC_U16 ? (const void*)(a.src_u16 + (size_t)k * np * 3)
                                       : SRC == SRC_F32 ? (const void*)(a.src_f32 + (size_t)k * np * 3) : (const void*)((const GS*)a.src_g + (size_t)k * np * 3);
        ss_row<SRC, GS, MODE == 0>(a, f, np, (EDGE ? lsb_reflect(y, H) : y) * W + xi0, o1, scale, v);
    };
    // a G_{l+1} row expanded along rows at the lane's pair (pyramid.rs:147)
    auto expand = [&](const float v[3], float2 e[3]) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const float l = __shfl_up_sync(ALL, v[c], 1), r = __shfl_down_sync(ALL, v[c], 1);
            e[c] = make_float2(lsb_exp_even(l, v[c], r), lsb_exp_odd(v[c], r));
        }
    };
    const int c0 = ((y0 - R) >> 1) + (ODD ? 2 : 1);  // the G_{l+1} row the first pair reads last
    float2 A[3], B[3], C[3];
    float ga[3], gb[3], gn[3];  // the next frame's first two G_{l+1} rows; the next row
    float2 va[3], vb[3];
    auto begin = [&](int k) {
        load_g1(k, scn, c0 - 2, ga);
        load_g1(k, scn, c0 - 1, gb);
        load_g1(k, scn, c0, gn);
        load_row(k, scn, y0 - R, va);
        load_row(k, scn, y0 - R + 1, vb);
    };
    begin(k0);
    int k = k0;
    float2 hs[2 * R + 1], L[R + 1][3];
    // one row: its values v (they become L), EXPAND's rows (three for an even row, two for an odd one)
    auto row = [&](const float2 v[3], int y, bool odd, const float2 E0[3], const float2 E1[3], const float2 E2[3], int j) {
#pragma unroll
        for (int q = 0; q < R; q++)
#pragma unroll
            for (int c = 0; c < 3; c++) L[q][c] = L[q + 1][c];
        float2 up[3];
#pragma unroll
        for (int c = 0; c < 3; c++) up[c] = odd ? exp_odd2(E1[c], E2[c]) : exp_even2(E0[c], E1[c], E2[c]);
        if (EDGE && (y < 0 || y >= H)) {
            // the reflected row's own neighbours and parity: y's, except in a level one row high, all of whose rows are row 0
            const int cy = lsb_reflect(y, H) >> 1;
            const bool from_odd = odd && H > 1;
            float t0[3], t1[3], t2[3];
            load_g1(k, sc, cy - 1, t0);
            load_g1(k, sc, cy, t1);
            load_g1(k, sc, cy + 1, t2);
            float2 D[3];
            if (!from_odd) expand(t0, up);
            expand(t1, D);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float l = __shfl_up_sync(ALL, t2[c], 1), r = __shfl_down_sync(ALL, t2[c], 1);
                const float2 F = make_float2(lsb_exp_even(l, t2[c], r), lsb_exp_odd(t2[c], r));
                up[c] = from_odd ? exp_odd2(D[c], F) : exp_even2(up[c], D[c], F);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            // the gain lane by lane: a packed product would be contracted into the packed subtraction
            L[R][c] = sub2(SRC == SRC_G ? v[c] : make_float2(__fmul_rn(v[c].x, gain[c]), __fmul_rn(v[c].y, gain[c])), up[c]);
        }
        float2 en;
        if (EDGE && a.use_chroma) {
            en = addl(addl(mul2(L[R][0], L[R][0]), mul2(L[R][1], L[R][1])), mul2(L[R][2], L[R][2]));
        } else {
            const float2 Y = luma2(L[R][0], L[R][1], L[R][2]);
            en = mul2(Y, Y);
        }
        // the window along rows
#pragma unroll
        for (int q = 0; q < 2 * R; q++) hs[q] = hs[q + 1];
        float2 h = en;
        if (R > 0) {
            if (EDGE) {  // the energies of columns beyond the level: the reflected ones'
                const int s0 = (xi0 - xb) & 63, s1 = (xi1 - xb) & 63;
                const float a0 = __shfl_sync(ALL, en.x, s0 >> 1), b0 = __shfl_sync(ALL, en.y, s0 >> 1);
                const float a1 = __shfl_sync(ALL, en.x, s1 >> 1), b1 = __shfl_sync(ALL, en.y, s1 >> 1);
                en = make_float2(s0 & 1 ? b0 : a0, s1 & 1 ? b1 : a1);
            }
            float e[2 + 2 * R];
            e[R] = en.x, e[R + 1] = en.y;
            e[R - 1] = __shfl_up_sync(ALL, en.y, 1);
            e[R + 2] = __shfl_down_sync(ALL, en.x, 1);
            if (R == 2) {
                e[0] = __shfl_up_sync(ALL, en.x, 1);
                e[2 * R + 1] = __shfl_down_sync(ALL, en.y, 1);
            }
            h = mul2(splat(binw<R>(0)), make_float2(e[0], e[1]));
#pragma unroll
            for (int q = 1; q <= 2 * R; q++) h = acc2<false>(h, binw<R>(q), make_float2(e[q], e[q + 1]));
        }
        hs[2 * R] = h;
        if (j < 0) return;
        // along columns, and the selection of row j
        float2 e = hs[0];
        if (R > 0) {
            e = mul2(splat(binw<R>(0)), hs[0]);
#pragma unroll
            for (int q = 1; q <= 2 * R; q++) e = acc2<false>(e, binw<R>(q), hs[q]);
        }
        float* p = st + 9 * 32 * j;
        if (EDGE && a.halo_mode) {
            const int yo = y0 + j;
            float wv[2] = {0.f, 0.f};
            if (lane >= 2 && lane < 30 && yo < H)
#pragma unroll
                for (int l = 0; l < 2; l++) {
                    if (xl + l >= W) continue;
                    float* hw = a.halo_w + (size_t)k * np + (size_t)yo * W + xl + l;
                    if (a.halo_mode == 1) *hw = halo_weight(l ? e.y : e.x, a.halo_p);
                    else wv[l] = *hw;
                }
            if (a.halo_mode == 2) {
                // halo control below the guide (fuse.rs:466-470): acc = L * w for the first frame, then acc += w * L;
                // best = the sum of the weights
#pragma unroll
                for (int l = 0; l < 2; l++) {
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const float m = __fmul_rn(wv[l], l ? L[0][c].y : L[0][c].x);
                        p[(2 * c + l) * 32] = k == 0 ? m : __fadd_rn(p[(2 * c + l) * 32], m);
                    }
                    p[(6 + l) * 32] = k == 0 ? wv[l] : __fadd_rn(p[(6 + l) * 32], wv[l]);
                }
                return;
            }
        }
#pragma unroll
        for (int l = 0; l < 2; l++) {
            const float ev = l ? e.y : e.x;
            if (ev > p[(6 + l) * 32]) {
                p[(6 + l) * 32] = ev;
#pragma unroll
                for (int c = 0; c < 3; c++) p[(2 * c + l) * 32] = l ? L[0][c].y : L[0][c].x;
                ((uint16_t*)(p + 8 * 32))[l] = (uint16_t)k;
            }
        }
    };
#pragma unroll 1
    for (; k < k1; k++) {
        expand(ga, B);
        expand(gb, C);
        sc = scn;
        if (SRC != SRC_G) {
            const int gon = a.xf[k].gain_on;
#pragma unroll
            for (int c = 0; c < 3; c++) gain[c] = (gon >> c) & 1 ? a.xf[k].gain[c] : 1.f;  // times 1: the value itself
        }
        if (k + 1 < k1) scn = make_float2(a.xf[k + 1].gscale, a.xf[k + 1].ginv);
#pragma unroll 1
        for (int p = 0; p < NP; p++) {
            const int y = y0 - R + 2 * p, j = 2 * p - 2 * R;
#pragma unroll
            for (int c = 0; c < 3; c++) A[c] = B[c], B[c] = C[c];
            expand(gn, C);
            float2 ra[3], rb[3];
#pragma unroll
            for (int c = 0; c < 3; c++) ra[c] = va[c], rb[c] = vb[c];
            const bool ends = p + 1 == NP || (EDGE && y + 2 >= H + R);  // rows past the window's reach: nobody's
            if (!ends) {
                load_g1(k, sc, c0 + p + 1, gn);
                load_row(k, sc, y + 2, va);
                load_row(k, sc, y + 3, vb);
            } else if (k + 1 < k1) {
                begin(k + 1);
            }
            if (ODD) {
                row(ra, y, true, A, A, B, j);
                row(rb, y + 1, false, A, B, C, j + 1);
            } else {
                row(ra, y, false, A, B, C, j);
                row(rb, y + 1, true, B, B, C, j + 1);
            }
            if (EDGE && ends) break;
        }
    }
}

constexpr int SS_STATE = SS_H * 9;  // words of a lane's state
constexpr size_t SS_SMEM = sizeof(float) * SS_WARPS * SS_STATE * 32;

// One CTA's tiles.
template <int SRC, class GS, int R>
__device__ __forceinline__ void select_cta(const SelBatch& T, int cta, float* sm) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int ri = 0;
    while (ri + 1 < T.n && cta >= T.r[ri + 1].cta0) ri++;
    const SelBatch::Rect& rc = T.r[ri];
    const FoldArgs& a = T.a[rc.lv];
    const int G = rc.groups, per = SS_WARPS / G, g = wid % G, sub = wid / G;  // a CTA: `per` tiles one above the other
    const int ci = cta - rc.cta0, by = ci / rc.ntx, bx = ci - by * rc.ntx;
    const int x0 = rc.x0 + bx * SS_W, y0 = rc.y0 + (by * per + sub) * SS_H;
    const int W = a.W, H = a.H;
    const size_t np = (size_t)W * H;
    const bool live = y0 < rc.y1;
    const int k0 = a.sel_k0 + (a.sel_k1 - a.sel_k0) * g / G, k1 = a.sel_k0 + (a.sel_k1 - a.sel_k0) * (g + 1) / G;
    const int xl = x0 - 4 + 2 * lane;
    const bool own0 = live && lane >= 2 && lane < 30 && xl < rc.x1, own1 = own0 && xl + 1 < rc.x1;
    float* st = sm + wid * SS_STATE * 32 + lane;
#pragma unroll
    for (int j = 0; j < SS_H; j++) {
        float* p = st + 9 * 32 * j;
#pragma unroll
        for (int q = 0; q < 9; q++) p[q * 32] = q == 6 || q == 7 ? -1.f : 0.f;  // any energy (>= 0) beats -1: frame 0 fills the accumulator (fuse.rs:409-412)
        if (g == 0 && a.sel_k0 > 0 && y0 + j < rc.y1) {  // resume: the state the frames before left
            const size_t o = (size_t)(y0 + j) * W + xl;
#pragma unroll
            for (int l = 0; l < 2; l++) {
                if (!(l ? own1 : own0)) continue;
#pragma unroll
                for (int c = 0; c < 3; c++) p[(2 * c + l) * 32] = a.acc[c * np + o + l];
                p[(6 + l) * 32] = a.best[o + l];
                if (a.winner) ((uint16_t*)(p + 8 * 32))[l] = a.winner[o + l];
            }
        }
    }
    if (live) {
        // the columns x0 - 4 .. x0 + 59 and the rows y0 - R .. y0 + 7 + R, and the G_{l+1} ones EXPAND reads, inside
        const bool inner = x0 >= 4 && x0 + 60 <= W && (x0 >> 1) + 30 <= a.W1 && y0 >= 4 && y0 + SS_H + R <= H && (y0 >> 1) + 6 <= a.H1;
        const bool plain = inner && !a.use_chroma && a.halo_mode == 0;
        if (!plain) ss_frames<SRC, GS, R, 2>(a, k0, k1, x0, y0, lane, st);
        else if (SRC != SRC_U16 && rc.vec) ss_frames<SRC, GS, R, SRC == SRC_U16 ? 1 : 0>(a, k0, k1, x0, y0, lane, st);
        else ss_frames<SRC, GS, R, 1>(a, k0, k1, x0, y0, lane, st);
    }
    // the groups' states in order: the first holding the largest energy wins, and within it its first frame did. Warp g
    // of a tile merges and writes every G-th row
    if (G > 1) __syncthreads();
    st -= g * SS_STATE * 32;
#pragma unroll 1
    for (int j = g; j < SS_H; j += G) {
        if (y0 + j >= rc.y1) break;
        const size_t o = (size_t)(y0 + j) * W + xl;
#pragma unroll
        for (int l = 0; l < 2; l++) {
            const float* p = st + 9 * 32 * j;
            float e = p[(6 + l) * 32];
            for (int q = 1; q < G; q++) {
                const float* pq = st + (q * SS_STATE + 9 * j) * 32;
                const float eq = pq[(6 + l) * 32];
                if (eq > e) e = eq, p = pq;
            }
            if (!(l ? own1 : own0)) continue;
            a.best[o + l] = e;
#pragma unroll
            for (int c = 0; c < 3; c++) a.acc[c * np + o + l] = p[(2 * c + l) * 32];
            if (a.winner) a.winner[o + l] = ((const uint16_t*)(p + 8 * 32))[l];
        }
    }
}

// TURNS: a launch bounded to fewer CTAs than there is work for, which they take in turn. A kernel of its own, because
// with the loop around them the strips keep more in registers and spill their window for it (R = 2: 460 to 850 bytes
// a thread instead of 210 to 310).
template <int SRC, class GS, int R, bool TURNS>
__global__ void __launch_bounds__(SS_WARPS * 32, SS_CTAS) select_strip_kernel(const __grid_constant__ SelBatch T) {
    extern __shared__ float sm[];
    if (!TURNS) return select_cta<SRC, GS, R>(T, blockIdx.x, sm);
#pragma unroll 1
    for (int cta = blockIdx.x; cta < T.ctas; cta += gridDim.x) {
        select_cta<SRC, GS, R>(T, cta, sm);
        __syncthreads();  // the groups' states are merged
    }
}
