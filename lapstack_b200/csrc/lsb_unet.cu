// The learned warm start of the WLS depth solve (no counterpart in the
// reference): a 4-level U-Net, 32 base channels, BF16 weights and
// activations with FP32 accumulation, that maps the quarter-resolution
// (guide luma, raw DfF depth, confidence) to the WLS solution. Its output is
// the x0 of MG-PCG, which then runs to the same relative residual as the
// plain solve, so the network changes only how fast the solve gets there.
//
// Layout: activations NHWC bf16 with channels a multiple of 32; weights
// [tap][cout][cin] bf16 for the forward conv (FP32 masters, Adam moments).
// conv3x3_kernel is an implicit GEMM on the tensor cores (mma.sync
// m16n8k16 bf16 -> f32): a CTA owns 8x16 output pixels x NT output
// channels; per 32-channel input chunk it stages the 10x18 input halo and the
// 9 x NT x 32 weights in shared memory (rows padded to 40 bf16 so the
// fragment loads hit 32 distinct banks). The same kernel computes dX in the
// backward pass with the flipped, transposed weights. The input loader reads
// a layer's input straight from where it lives: the previous activation, a
// 2x2 average pool of a finer one (encoder), a nearest 2x upsample of a
// coarser one (decoder), and the channel concat of an upsampled tensor with
// a skip tensor, so no pooled, upsampled or concatenated copy is written.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "lapstack_b200.h"
#include "lsb_common.cuh"

namespace lsb {

constexpr int UN_CH = 32;        // input-chunk channels
constexpr int UN_TH = 8, UN_TW = 16;  // output tile (pixels)
constexpr int UN_HP = UN_TH + 2, UN_WP = UN_TW + 2;
constexpr int UN_LD = UN_CH + 8;  // padded row (bf16)
constexpr int UN_THREADS = 128;

enum { SRC_SAME = 0, SRC_UP = 1, SRC_POOL = 2 };

struct ConvArgs {
    const __nv_bfloat16* src1;
    const __nv_bfloat16* src2;
    int c1, c1s, mode1;  // channels of source 1 read, its channel stride, its mode
    int c2s, mode2;      // source 2 (channels c1..cin-1), its channel stride
    int cin, cout;
    const __nv_bfloat16* w;  // [9][cout][cin]
    const __nv_bfloat16* wp;  // the same packed for the tcgen05 path: [cout / N][cin / 32][9][4][N][8]
    const float* bias;       // [cout] or null
    int relu;
    __nv_bfloat16* out;      // [B][H][W][cout] bf16, or null
    float* out_f32;          // [B][H][W][cout] f32, or null
    float* out_c0;           // [B][H][W] channel 0 only (f32), or null
    int B, H, W;             // output grid
};

__device__ __forceinline__ uint32_t bf2_as_u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }

// 8 consecutive channels (16 bytes) of one input pixel, through the source's mode.
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* src, int cs, int mode, int b, int y, int x, int H, int W, int c) {
    if (mode == SRC_SAME) {
        return *reinterpret_cast<const uint4*>(src + (((size_t)b * H + y) * W + x) * cs + c);
    }
    if (mode == SRC_UP) {
        const int h2 = H >> 1, w2 = W >> 1;
        return *reinterpret_cast<const uint4*>(src + (((size_t)b * h2 + (y >> 1)) * w2 + (x >> 1)) * cs + c);
    }
    // SRC_POOL: the mean of the 2x2 block of the finer source
    const int H2 = H * 2, W2 = W * 2;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] = 0.f;
#pragma unroll
    for (int dy = 0; dy < 2; dy++)
#pragma unroll
        for (int dx = 0; dx < 2; dx++) {
            uint4 v = *reinterpret_cast<const uint4*>(src + (((size_t)b * H2 + 2 * y + dy) * W2 + 2 * x + dx) * cs + c);
            const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float2 f = __bfloat1622float2(p[i]);
                acc[2 * i] += f.x;
                acc[2 * i + 1] += f.y;
            }
        }
    uint4 o;
    __nv_bfloat162* q = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int i = 0; i < 4; i++) q[i] = __floats2bfloat162_rn(acc[2 * i] * 0.25f, acc[2 * i + 1] * 0.25f);
    return o;
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// out[p][n] = sum_{tap, ci} X[p + off(tap)][ci] * w[tap][n][ci] (+ bias, ReLU), zero padding.
template <int NT>
__global__ void __launch_bounds__(UN_THREADS) conv3x3_kernel(const ConvArgs a) {
    extern __shared__ __align__(16) unsigned char un_smem[];
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(un_smem);  // [UN_HP*UN_WP][UN_LD]
    __nv_bfloat16* ws = xs + UN_HP * UN_WP * UN_LD;                  // [9][NT][UN_LD]
    const int tiles_x = (a.W + UN_TW - 1) / UN_TW;
    const int x0 = (blockIdx.x % tiles_x) * UN_TW, y0 = (blockIdx.x / tiles_x) * UN_TH;
    const int n0 = blockIdx.y * NT, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    constexpr int NJ = NT / 8;
    float acc[2][NJ][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int j = 0; j < NJ; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[m][j][q] = 0.f;

    for (int c0 = 0; c0 < a.cin; c0 += UN_CH) {
        const bool first = c0 < a.c1;
        const __nv_bfloat16* src = first ? a.src1 : a.src2;
        const int cs = first ? a.c1s : a.c2s, mode = first ? a.mode1 : a.mode2, cb = first ? c0 : c0 - a.c1;
        // stage the input halo: UN_HP*UN_WP pixels x 4 vectors of 8 channels
        for (int i = tid; i < UN_HP * UN_WP * 4; i += UN_THREADS) {
            const int pix = i >> 2, v = i & 3;
            const int yy = y0 - 1 + pix / UN_WP, xx = x0 - 1 + pix % UN_WP;
            uint4 val = make_uint4(0u, 0u, 0u, 0u);
            if (yy >= 0 && yy < a.H && xx >= 0 && xx < a.W) val = load8(src, cs, mode, b, yy, xx, a.H, a.W, cb + 8 * v);
            *reinterpret_cast<uint4*>(xs + pix * UN_LD + 8 * v) = val;
        }
        // stage the weights of this chunk: 9 x NT rows of 32 channels
        for (int i = tid; i < 9 * NT * 4; i += UN_THREADS) {
            const int row = i >> 2, v = i & 3;
            const int tap = row / NT, n = row % NT;
            const uint4 val = *reinterpret_cast<const uint4*>(a.w + ((size_t)tap * a.cout + n0 + n) * a.cin + c0 + 8 * v);
            *reinterpret_cast<uint4*>(ws + row * UN_LD + 8 * v) = val;
        }
        __syncthreads();
#pragma unroll 1
        for (int tap = 0; tap < 9; tap++) {
            const int ky = tap / 3, kx = tap % 3;
#pragma unroll
            for (int kk = 0; kk < UN_CH; kk += 16) {
                uint32_t af[2][4];
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const int r = 2 * warp + m;  // tile row of this m16 block
                    const __nv_bfloat16* p0 = xs + ((r + ky) * UN_WP + g + kx) * UN_LD + kk + 2 * t;
                    const __nv_bfloat16* p1 = p0 + 8 * UN_LD;
                    af[m][0] = *reinterpret_cast<const uint32_t*>(p0);
                    af[m][1] = *reinterpret_cast<const uint32_t*>(p1);
                    af[m][2] = *reinterpret_cast<const uint32_t*>(p0 + 8);
                    af[m][3] = *reinterpret_cast<const uint32_t*>(p1 + 8);
                }
#pragma unroll
                for (int j = 0; j < NJ; j++) {
                    const __nv_bfloat16* q = ws + (tap * NT + 8 * j + g) * UN_LD + kk + 2 * t;
                    const uint32_t b0 = *reinterpret_cast<const uint32_t*>(q);
                    const uint32_t b1 = *reinterpret_cast<const uint32_t*>(q + 8);
                    mma_bf16(acc[0][j], af[0][0], af[0][1], af[0][2], af[0][3], b0, b1);
                    mma_bf16(acc[1][j], af[1][0], af[1][1], af[1][2], af[1][3], b0, b1);
                }
            }
        }
        __syncthreads();
    }
    // epilogue: c0,c1 -> (pixel g, channels 2t, 2t+1); c2,c3 -> pixel g+8
#pragma unroll
    for (int m = 0; m < 2; m++) {
        const int y = y0 + 2 * warp + m;
        if (y >= a.H) continue;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int x = x0 + g + 8 * half;
            if (x >= a.W) continue;
            const size_t pix = ((size_t)b * a.H + y) * a.W + x;
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const int n = n0 + 8 * j + 2 * t;
                float v0 = acc[m][j][2 * half], v1 = acc[m][j][2 * half + 1];
                if (a.bias) {
                    v0 += a.bias[n];
                    v1 += a.bias[n + 1];
                }
                if (a.relu) {
                    v0 = fmaxf(v0, 0.f);
                    v1 = fmaxf(v1, 0.f);
                }
                if (a.out) *reinterpret_cast<__nv_bfloat162*>(a.out + pix * a.cout + n) = __floats2bfloat162_rn(v0, v1);
                if (a.out_f32) *reinterpret_cast<float2*>(a.out_f32 + pix * a.cout + n) = make_float2(v0, v1);
                if (a.out_c0 && n == 0) a.out_c0[pix] = v0;
            }
        }
    }
}

// ------------------------------------------------- the same conv on tcgen05
// conv3x3_tc_kernel: the implicit GEMM on the 5th-generation tensor cores. A tile is 16 x 8 output pixels
// (M = 128, one TMEM lane per pixel) x N output channels (one fp32 TMEM column each); cin goes by chunks of
// 32. The operands lie in shared memory in the canonical no-swizzle K-major layout of the UMMA descriptors
// (8 rows of 16 bytes per core matrix): the 18 x 10 halo of a chunk as [k8][pixel][8 channels], so that the
// tap (ky, kx) of the A operand is the same layout started (ky * 10 + kx) pixels later (rows of 8 pixels 10
// pixels apart: SBO = 160 B, the next 8 channels LBO = one plane further); the weights as [tap][k8][n][8],
// which is how cast_weights_kernel packs them, so that a chunk's weights are one bulk copy.
// One persistent CTA per SM, its warps split by role: up to eight load halos into two rings of stages, the
// even and the odd tiles' (cp.async, zero-filled outside the image; a pooled source by registers), one thread
// copies weights, two warps issue 9 taps x 2 K-steps of tcgen05.mma (kind::f16, BF16 x BF16 -> FP32) per tile
// and chunk, the even tiles and the odd ones, and commit them to mbarriers, two sets of four warps read finished
// accumulators (tcgen05.ld, a lane quarter each), add the bias, apply ReLU and store NHWC while the next tiles
// multiply: the TMEM holds 4 or 8 accumulators. Every product is added in the order chunk, tap, K-step.
// A layer whose weights fit the weight buffers (two chunks, four at N = 32) keeps them for the whole launch and
// takes its tiles one by one; a larger one streams them, chunk by chunk, over groups of as many tiles as
// there are accumulators.
// What bounds it: an MMA of M = 128, K = 16 reads 4 KB of A from shared memory, 32 cycles, whatever N is, so a
// tile and chunk takes 576 cycles at least; measured 1300 to 1500 at N = 32, where each role's own instructions
// (about 130 a tile in the epilogue, 330 a halo in a loader) are what is left, 3 TB/s. One MMA warp instead of
// two took 1800, one set of epilogue warps 1600, MMAs issued by one divergent lane 2400 (56 cycles each to move
// their operands to the uniform registers). The 15 layers on a 2064 x 1376 grid (1.02 TFLOP): 3.7 ms as CTAs of
// one tile that staged, multiplied and stored in turn, 1.55 ms here.
constexpr int TC_TH = 16, TC_TW = 8;
constexpr int TC_HP = TC_TH + 2, TC_WP = TC_TW + 2, TC_PIX = TC_HP * TC_WP;  // 18 x 10 halo
// try_wait polls per wait: far beyond a chunk's MMAs (microseconds); a CTA that meets a set error word
// (an earlier wait ran out) does nothing
constexpr unsigned TC_SPIN_LIMIT = 1u << 20;

constexpr int TC_PLANE = TC_PIX * 16 + 32;  // bytes of 8 channels of a halo (+32: bank spread of the stores)
constexpr int TC_STAGE = 4 * TC_PLANE;      // a chunk's halo
// The warps of a CTA by role. Warp w issues on scheduler w % 4: the two MMA warps (which take the tiles in
// turn, so that one's waits and commits hide behind the other's MMAs) share theirs with little else.
constexpr int TC_EW = 4;                                // 0-3, 12-15: the epilogue of the even and the odd tiles, a TMEM lane quarter each
constexpr int TC_MMA0 = 4, TC_MMA1 = 5, TC_WW = 8;      // the MMAs, the weights
constexpr int TC_LW = 8;                                // 6, 7, 9-11, 17-19: the loaders
__device__ __forceinline__ int tc_loader(int w) { return w < 6 || w == 8 || (w > 11 && w < 17) ? -1 : w > 16 ? w - 12 : w - 6 - (w > 8); }
constexpr int TC_THREADS = 32 * 20;
__host__ __device__ constexpr int tc_chunk(int n) { return 9 * 4 * n * 16; }
__host__ __device__ constexpr int tc_wbufs(int n) { return n == 32 ? 4 : 2; }  // weight buffers (chunks)
// accumulators in TMEM: even, so that each belongs to the even or to the odd tiles (a wait by parity then never
// meets a phase of the other role's)
__host__ __device__ constexpr int tc_accs(int n) { return n >= 96 ? 4 : 8; }
__host__ __device__ constexpr int tc_depth(int n) { return n == 128 ? 6 : n == 96 ? 8 : 12; }  // halos, in two rings
__host__ __device__ constexpr size_t tc_smem(int n) {
    return (size_t)tc_wbufs(n) * tc_chunk(n) + tc_depth(n) * TC_STAGE + 8 * (2 * tc_depth(n) + 2 * 4 + 2 * 8 + 2) + 16 + 4 * n;
}
static_assert(tc_smem(32) <= 227 * 1024 && tc_smem(64) <= 227 * 1024 && tc_smem(96) <= 227 * 1024 && tc_smem(128) <= 227 * 1024,
              "shared memory");

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// the UMMA shared-memory descriptor, no swizzle (layout type 0), version 1; addresses and offsets in bytes
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) |
           (1ull << 46);
}
// the instruction descriptor of kind::f16: D f32, A and B bf16, both K-major, M = 128, N
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    uint32_t done = 0;
    for (unsigned it = 0; it < TC_SPIN_LIMIT && !done; it++)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
    return done != 0;
}
__device__ __forceinline__ void umma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// The output channels one CTA takes (N): the largest of 128, 96, 64 and 32 that divides cout.
__host__ __device__ constexpr int tc_block(int cout) {
    return cout % 128 == 0 ? 128 : cout % 96 == 0 ? 96 : cout % 64 == 0 ? 64 : cout % 32 == 0 ? 32 : 0;
}
// A bounded wait that also gives up once another role of the CTA has. A poll may suspend the warp for up to
// TC_WAIT_NS, so that waiting warps do not crowd the shared-memory pipe the others work through.
constexpr unsigned TC_WAIT_NS = 1000;
__device__ __forceinline__ bool mbar_wait_or(uint32_t bar, uint32_t parity, volatile int* abort) {
    uint32_t done = 0;
    for (unsigned it = 0; it < TC_SPIN_LIMIT; it++) {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(done)
                     : "r"(bar), "r"(parity), "r"(TC_WAIT_NS)
                     : "memory");
        if (done) return true;
        if (*abort) return false;
    }
    *abort = 1;
    return false;
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}
// 32 bytes in one store (whole sectors)
__device__ __forceinline__ void st32(void* p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                 "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

// A CTA's tiles, one gridDim.x apart, walked without divisions.
struct TileWalk {
    int b, ty, tx;
    __device__ __forceinline__ void step(int sb, int sy, int sx, int tiles_y, int tiles_x) {
        tx += sx;
        if (tx >= tiles_x) tx -= tiles_x, ty++;
        ty += sy;
        if (ty >= tiles_y) ty -= tiles_y, b++;
        b += sb;
    }
};

template <int N>
__global__ void __launch_bounds__(TC_THREADS, 1) conv3x3_tc_kernel(const ConvArgs a, int* status) {
    extern __shared__ __align__(128) unsigned char tc_smem_[];
    constexpr int NB = tc_wbufs(N), NACC = tc_accs(N), CB = tc_chunk(N), DEPTH = tc_depth(N);
    unsigned char* Ws = tc_smem_;
    unsigned char* As = tc_smem_ + NB * CB;
    uint64_t* bars = reinterpret_cast<uint64_t*>(As + DEPTH * TC_STAGE);
    constexpr int RING = DEPTH / 2;  // halos of the even tiles, then of the odd ones: one consumer each
    const uint32_t a_full = smem_u32(bars), a_empty = a_full + 8 * DEPTH, w_full = a_empty + 8 * DEPTH, w_empty = w_full + 32,
                   d_full = w_empty + 32, d_empty = d_full + 64, fin = d_empty + 64;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2 * DEPTH + 26);
    volatile int* abort = reinterpret_cast<volatile int*>(tslot + 1);
    float* bs = reinterpret_cast<float*>(bars + 2 * DEPTH + 28);  // the bias
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles_x = (a.W + TC_TW - 1) / TC_TW, tiles_y = (a.H + TC_TH - 1) / TC_TH, ntiles = tiles_x * tiles_y * a.B;
    const int nloc = (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // this CTA's tiles
    const int n0 = blockIdx.y * N, nch = a.cin / UN_CH;
    const bool resident = nch <= NB;
    const int G = resident ? 1 : NACC;
    if (__syncthreads_or(*(volatile int*)status)) return;  // an earlier CTA's wait ran out: nothing is allocated yet
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int q = 0; q < DEPTH; q++) mbar_init(a_full + 8 * q, 1), mbar_init(a_empty + 8 * q, 1);
        for (int q = 0; q < 4; q++) mbar_init(w_full + 8 * q, 1), mbar_init(w_empty + 8 * q, 2);
        for (int q = 0; q < 8; q++) mbar_init(d_full + 8 * q, 1), mbar_init(d_empty + 8 * q, TC_EW);
        mbar_init(fin, 1), mbar_init(fin + 8, 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    for (int q = tid; q < N; q += TC_THREADS) bs[q] = a.bias ? a.bias[n0 + q] : 0.f;
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);
    // The next kernel may start its CTAs where these leave room; what the kernel before wrote is read, and what it may
    // still read is written, only behind the wait. The weights and biases it does not write: their copy starts at once.
    asm volatile("griddepcontrol.launch_dependents;");
    if (warp != TC_WW) asm volatile("griddepcontrol.wait;" ::: "memory");
    const int sx = (int)gridDim.x % tiles_x, sy = (int)gridDim.x / tiles_x % tiles_y, sb = (int)gridDim.x / (tiles_x * tiles_y);
    TileWalk at{(int)blockIdx.x / (tiles_x * tiles_y), (int)blockIdx.x / tiles_x % tiles_y, (int)blockIdx.x % tiles_x};
    if (const int lw = tc_loader(warp); lw >= 0) {
        // ---- the loaders, half of them for each ring (the even and the odd tiles): a warp takes every LW-th halo of
        // its ring, 180 pixels x 4 vectors of 8 channels: lane l the vector l % 4 of the pixels l / 4, l / 4 + 8, ...
        constexpr int Q = (TC_PIX + 7) / 8;
        // a warp waits for its slot by parity, having last seen the halo LW + RING back consumed: with LW > RING
        // the slot could be two phases behind, which a parity cannot tell from free
        constexpr int LW = TC_LW / 2 < RING ? TC_LW / 2 : RING;
        static_assert(LW <= RING, "a loader warp's stride");
        const int ring = lw & 1;
        const int v = lane & 3, pix0 = lane >> 2;
        int seq = 0, held = -1;
        bool ok = lw / 2 < LW;
        auto hand_over = [&]() {  // the copies into slot `held` are done: visible to the tensor cores, then full
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(a_full + 8 * held);
        };
        for (int k0 = 0; k0 < nloc && ok; k0 += G) {
            const int gn = min(G, nloc - k0);
            TileWalk t = at;
            for (int ch = 0; ch < nch && ok; ch++) {
                const int c0 = ch * UN_CH;
                const bool first = c0 < a.c1;
                const int cs = first ? a.c1s : a.c2s, mode = first ? a.mode1 : a.mode2;
                const int up = mode == SRC_UP ? 1 : 0, hs = a.H >> up, ws = a.W >> up;
                const __nv_bfloat16* src = (first ? a.src1 : a.src2) + (first ? c0 : c0 - a.c1) + 8 * v;
                t = at;
                for (int g = 0; g < gn; g++, t.step(sb, sy, sx, tiles_y, tiles_x)) {
                    if (((k0 + g) & 1) != ring) continue;
                    const int mine = seq++;  // this halo's place in its ring's order
                    if (mine % LW != lw / 2) continue;
                    const int st = ring * RING + mine % RING;
                    if (held >= 0) {
                        asm volatile("cp.async.wait_group 0;" ::: "memory");
                        hand_over();
                    }
                    if (mine >= RING) ok = mbar_wait_or(a_empty + 8 * st, (uint32_t)((mine / RING - 1) & 1), abort);
                    ok = __all_sync(0xffffffffu, ok);
                    held = -1;
                    if (!ok) break;
                    unsigned char* S = As + st * TC_STAGE + v * TC_PLANE + pix0 * 16;
                    const int yb = t.ty * TC_TH - 1, xb = t.tx * TC_TW - 1;
                    int c = pix0, y = yb;  // pixel pix0 of the halo: row 0, column pix0 (pix0 < 8 < TC_WP)
                    if (mode == SRC_POOL) {
#pragma unroll 4
                        for (int q = 0; q < Q; q++) {
                            const int x = xb + c;
                            uint4 val = make_uint4(0u, 0u, 0u, 0u);
                            if ((unsigned)y < (unsigned)a.H && (unsigned)x < (unsigned)a.W) val = load8(src, cs, SRC_POOL, t.b, y, x, a.H, a.W, 0);
                            if (8 * q + pix0 < TC_PIX) *reinterpret_cast<uint4*>(S + q * 128) = val;
                            c += 8;
                            if (c >= TC_WP) c -= TC_WP, y++;
                        }
                    } else {
                        const __nv_bfloat16* img = src + (size_t)t.b * hs * ws * cs;
                        const uint32_t d0 = smem_u32(S);
#pragma unroll
                        for (int q = 0; q < Q; q++) {
                            const int x = xb + c;
                            const bool in = (unsigned)y < (unsigned)a.H && (unsigned)x < (unsigned)a.W;
                            const __nv_bfloat16* p = in ? img + ((size_t)(y >> up) * ws + (x >> up)) * cs : src;
                            if (8 * q + pix0 < TC_PIX)
                                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d0 + q * 128), "l"(p), "r"(in ? 16 : 0)
                                             : "memory");
                            c += 8;
                            if (c >= TC_WP) c -= TC_WP, y++;
                        }
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    held = st;
                }
            }
            at = t;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (ok && held >= 0) hand_over();
    } else if (warp == TC_WW) {
        // ---- the weights: one bulk copy per chunk; the resident ones once
        if (lane == 0) {
            const unsigned char* wp = reinterpret_cast<const unsigned char*>(a.wp) + (size_t)blockIdx.y * nch * CB;
            const int total = resident ? nch : nch * ((nloc + G - 1) / G);
            int seq = 0;
            for (; seq < total; seq++) {
                const int buf = seq % NB;
                if (seq >= NB && !mbar_wait_or(w_empty + 8 * buf, (uint32_t)((seq / NB - 1) & 1), abort)) break;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(w_full + 8 * buf), "r"(CB) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 smem_u32(Ws + buf * CB)),
                             "l"(wp + (size_t)(seq % nch) * CB), "r"(CB), "r"(w_full + 8 * buf)
                             : "memory");
            }
            for (int q = max(0, seq - NB); q < seq; q++) mbar_wait(w_full + 8 * (q % NB), (uint32_t)((q / NB) & 1));  // none left in flight
        }
    } else if (warp == TC_MMA0 || warp == TC_MMA1) {
        // ---- the MMAs: 9 taps x 2 K-steps per tile and chunk. The whole warp walks the loop, so that descriptors
        // and addresses stay warp-uniform (issued from one divergent lane, every operand of every MMA is moved
        // to the uniform registers by itself: 56 cycles an MMA); one elected lane issues.
        constexpr uint32_t IDESC = umma_idesc_bf16(N);
        const bool leader = elect_one();
        const uint64_t da0 = umma_desc(smem_u32(As), TC_PLANE, TC_WP * 16), db0 = umma_desc(smem_u32(Ws), N * 16, 8 * 16);
        int st = 0, buf = 0;
        const int mw = warp - TC_MMA0;
        uint32_t aph = 0, wph = 0;
        bool ok = true;
        for (int k0 = 0; k0 < nloc && ok; k0 += G) {
            const int gn = min(G, nloc - k0);
            for (int ch = 0; ch < nch && ok; ch++) {
                if (resident) buf = ch;
                if (!resident || k0 == 0) ok = mbar_wait_or(w_full + 8 * buf, wph, abort);
                const uint64_t dbc = db0 + (uint32_t)(buf * (CB >> 4));
                for (int g = 0; g < gn && ok; g++) {
                    const int k = k0 + g, acc = k % NACC;
                    if ((k & 1) != mw) continue;  // the other MMA warp's tile
                    if (ch == 0 && k >= NACC) ok = mbar_wait_or(d_empty + 8 * acc, (uint32_t)((k / NACC - 1) & 1), abort);
                    const int slot = mw * RING + st;
                    ok = ok && mbar_wait_or(a_full + 8 * slot, aph, abort);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint64_t dac = da0 + (uint32_t)(slot * (TC_STAGE >> 4));
                    const uint32_t d = tmem + acc * N;
                    if (leader) {
#pragma unroll
                        for (int tap = 0; tap < 9; tap++)
#pragma unroll
                            for (int j = 0; j < 2; j++)
                                umma_bf16(d, dac + ((2 * j * TC_PLANE) >> 4) + (tap / 3) * TC_WP + tap % 3, dbc + (tap * 4 + 2 * j) * N, IDESC,
                                          (tap > 0 || j > 0) ? 1u : ch > 0);
                        umma_commit(a_empty + 8 * slot);
                        if (ch == nch - 1) umma_commit(d_full + 8 * acc);
                    }
                    __syncwarp();
                    if (++st == RING) st = 0, aph ^= 1;
                }
                if (!resident) {  // this warp's MMAs on the chunk's weights, if any
                    if (ok && leader) umma_commit(w_empty + 8 * buf);
                    if (++buf == NB) buf = 0, wph ^= 1;
                }
            }
        }
        if (!ok) {  // the MMAs in flight get a bounded wait before the TMEM goes
            if (leader) umma_commit(fin + 8 * mw);
            __syncwarp();
            mbar_wait(fin + 8 * mw, 0);
        }
    } else if (warp < TC_EW || (warp >= 12 && warp < 16)) {
        // ---- the epilogue: pixel m = 32 quarter + lane = (row m / 8, column m % 8)
        const int quarter = warp & 3, m = 32 * quarter + lane, set = warp >= 12;
        bool ok = true;
        for (int k = 0; k < nloc && ok; k++, at.step(sb, sy, sx, tiles_y, tiles_x)) {
            if ((k & 1) != set) continue;
            const int acc = k % NACC;
            ok = __all_sync(0xffffffffu, mbar_wait_or(d_full + 8 * acc, (uint32_t)((k / NACC) & 1), abort));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const int y = at.ty * TC_TH + m / TC_TW, x = at.tx * TC_TW + m % TC_TW;
            const bool in = y < a.H && x < a.W;
            const size_t pix = ((size_t)at.b * a.H + y) * a.W + x;
#pragma unroll 1
            for (int c = 0; c < N; c += 32) {
                __syncwarp();  // lanes outside the image skip the stores below; the read is the whole warp's
                uint32_t r[32];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                    "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                      "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
                      "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                      "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                    : "r"(tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(acc * N + c)));
                asm volatile("tcgen05.wait::ld.sync.aligned;");
                if (c + 32 == N) {  // the accumulator is read: the next tile may take it
                    asm volatile("tcgen05.fence::before_thread_sync;");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty + 8 * acc);
                }
                if (!in) continue;
                const int n = n0 + c;
                if (a.bias) {
#pragma unroll
                    for (int q = 0; q < 32; q += 4) {
                        const float4 b4 = *reinterpret_cast<const float4*>(bs + c + q);
                        r[q] = __float_as_uint(__uint_as_float(r[q]) + b4.x);
                        r[q + 1] = __float_as_uint(__uint_as_float(r[q + 1]) + b4.y);
                        r[q + 2] = __float_as_uint(__uint_as_float(r[q + 2]) + b4.z);
                        r[q + 3] = __float_as_uint(__uint_as_float(r[q + 3]) + b4.w);
                    }
                }
                if (a.relu) {
#pragma unroll
                    for (int q = 0; q < 32; q++) r[q] = __float_as_uint(fmaxf(__uint_as_float(r[q]), 0.f));
                }
                if (a.out_c0 && n == 0) a.out_c0[pix] = __uint_as_float(r[0]);
                if (a.out) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t o[8];
#pragma unroll
                        for (int q = 0; q < 8; q++)
                            o[q] = bf2_as_u32(__floats2bfloat162_rn(__uint_as_float(r[16 * h + 2 * q]), __uint_as_float(r[16 * h + 2 * q + 1])));
                        st32(a.out + pix * a.cout + n + 16 * h, o);
                    }
                }
                if (a.out_f32) {
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        uint32_t o[8];
#pragma unroll
                        for (int q = 0; q < 8; q++) o[q] = r[8 * h + q];
                        st32(a.out_f32 + pix * a.cout + n + 8 * h, o);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (tid == 0 && *abort) atomicOr(status, 0x100);  // a wait ran out: the output is not whole
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------ backward parts
// One user of a tensor in the backward pass: the dX of the layer that read it (at that layer's grid H x W,
// cin channels, the tensor's from coff on) and how that layer read it.
struct GradUse {
    const float* dx;
    int cin, coff, mode, H, W;
};
__device__ __forceinline__ void ld8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
// dZ of a layer's output tensor (Hs x Ws, C channels), rounded to bf16 (the operand of the dX conv and dW): the
// gradients its one or two users send back -- SAME adds, UP sums the 4 children of a coarse pixel, POOL spreads
// 1/4 -- masked by the ReLU (Y > 0). One thread per 8 channels of a pixel, 16 to 32 bytes per access, each tensor
// read and written once: routing each dX into an FP32 gradient and masking that took three passes with one value
// a thread (1.57 ms of a step of 8 crops of 256 x 256, their clearing included; 0.25 ms here, HBM-bound).
__global__ void grad_gather_kernel(GradUse u0, GradUse u1, int uses, const __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ dz, int Hs,
                                   int Ws, int C, size_t items, int relu) {
    const int cv = C / 8;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < items; i += (size_t)gridDim.x * blockDim.x) {
        const size_t p = i / cv;
        const int c = (int)(i - p * cv) * 8;
        const size_t row = p / Ws;
        const int px = (int)(p - row * Ws), b = (int)(row / Hs), py = (int)(row - (size_t)b * Hs);
        float g[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (k >= uses) break;
            const GradUse& u = k ? u1 : u0;
            const float* dx = u.dx + u.coff + c;
            float v[8];
            if (u.mode == SRC_SAME) {
                ld8(dx + p * u.cin, v);
            } else if (u.mode == SRC_UP) {
                float w[4][8];
#pragma unroll
                for (int q = 0; q < 4; q++) ld8(dx + (((size_t)b * u.H + 2 * py + q / 2) * u.W + 2 * px + q % 2) * u.cin, w[q]);
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = w[0][e] + w[1][e] + w[2][e] + w[3][e];
            } else {
                ld8(dx + (((size_t)b * u.H + py / 2) * u.W + px / 2) * u.cin, v);
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] *= 0.25f;
            }
#pragma unroll
            for (int e = 0; e < 8; e++) g[e] += v[e];
        }
        if (relu) {
            const uint4 yv = *reinterpret_cast<const uint4*>(y + p * C + c);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&yv);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 f = __bfloat1622float2(h[e]);
                if (!(f.x > 0.f)) g[2 * e] = 0.f;
                if (!(f.y > 0.f)) g[2 * e + 1] = 0.f;
            }
        }
        uint4 o;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int e = 0; e < 4; e++) h[e] = __floats2bfloat162_rn(g[2 * e], g[2 * e + 1]);
        *reinterpret_cast<uint4*>(dz + p * C + c) = o;
    }
}
// the output layer: only channel 0 of its 32 carries a gradient
__global__ void out_grad_kernel(const float* __restrict__ dy0, __nv_bfloat16* __restrict__ dz, size_t npx) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npx * 4; i += (size_t)gridDim.x * blockDim.x) {
        uint4 o = make_uint4(0u, 0u, 0u, 0u);
        if (i % 4 == 0) o.x = __bfloat16_as_ushort(__float2bfloat16_rn(dy0[i / 4]));
        reinterpret_cast<uint4*>(dz)[i] = o;
    }
}

// dW[tap][co][ci] = sum over pixels of dZ[p][co] X[p + off(tap)][ci], and db[co] = sum of dZ, on the
// 5th-generation tensor cores: a GEMM whose K is the pixels. A CTA owns CO couts x 32 cins and every
// splits-th 16 x 8 pixel tile. A tile's sums are made in TMEM (D: a lane per cout, a column per (tap, cin)) and
// added, tile by tile, to FP32 registers, rounded to nearest; a CTA's sums go out once, as vector reductions. (The
// tensor core's own accumulator drops what lies below its last place at every step, so sums of positive products left in
// it over all of a CTA's tiles fell short in proportion to their number: by 7.8e-6 on 8 crops of 256 x 256 and 2.4e-5
// on 1024 x 1024; here by less than 5e-8, for 0.1 ms a step of those crops.) Both operands are MN-major (the channel is
// contiguous in a pixel): A = dZ as [c8][pixel][8 channels], B = X's halo in three copies, one per kx,
// as [kx][c8][18 rows][8 pixels][8 channels], so that one MMA takes the three kx of a ky (N = 96) and ky
// is a start address one row further down. db is one more column block whose B is all ones.
// What bounds it: an MMA of M = 128, K = 16 reads 4 KB of A from shared memory whatever its N, so
// 24 MMAs a tile (N = 96) instead of 72 (N = 32) is what the three copies buy; the rest is staging
// (20 to 43 KB a tile), prefetched into registers one tile ahead and double-buffered against the MMAs.
// Couts below 128 leave lanes that hold products of whatever lies behind A's planes (in bounds; a
// lane's sums never mix with another's); they are not read.
// Measured over the 15 layers of a step of 8 crops of 256 x 256: 13.4 ms as register sums on the CUDA
// cores, 0.90 ms here (0.17 TFLOP: 190 TFLOP/s), of which the reads of the TMEM 0.10.
constexpr int DW_THREADS = 256;
constexpr int DW_XROWS = TC_HP * TC_TW;                     // 144 pixels of one copy of X
constexpr int DW_XPLANE = DW_XROWS * 16 + 32;               // bytes of 8 channels of one copy (+32: bank spread)
constexpr int DW_XBYTES = 12 * DW_XPLANE;                   // 3 copies x 4 planes
constexpr int DW_ZPX = TC_TH * TC_TW;                       // 128 pixels of dZ
__host__ __device__ constexpr int dw_zplane(int co) { return DW_ZPX * 16 + (co == 32 ? 32 : 16); }
// one stage: dZ's planes, then X's; A's 16 planes of an M = 128 operand end inside the stage for every co
__host__ __device__ constexpr int dw_stage(int co) { return (co / 8 * dw_zplane(co) + DW_XBYTES + 127) / 128 * 128; }
__host__ __device__ constexpr size_t dw_smem_bytes(int co) { return (size_t)2 * dw_stage(co) + 512 + 32; }
static_assert(dw_stage(32) >= 16 * dw_zplane(32) && dw_stage(64) >= 16 * dw_zplane(64) && dw_stage(128) >= 16 * dw_zplane(128),
              "A's planes stay inside the stage");
constexpr uint32_t DW_COLS = 512, DW_DB_COL = 288;
constexpr int DW_BLOCKS = DW_DB_COL / 16 / 2;  // blocks of 16 columns a warp reads

__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <int CO>
__global__ void __launch_bounds__(DW_THREADS, 1) conv_dw_kernel(const ConvArgs a, const __nv_bfloat16* __restrict__ dz,
                                                                float* __restrict__ dw, float* __restrict__ db, int* status) {
    extern __shared__ __align__(128) unsigned char dw_smem[];
    constexpr int ZP = dw_zplane(CO), STAGE = dw_stage(CO), ZV = CO / 8, ZQ = DW_ZPX * ZV / DW_THREADS;
    constexpr int XU = TC_PIX * 4, XQ = (XU + DW_THREADS - 1) / DW_THREADS;
    unsigned char* ones = dw_smem + 2 * STAGE;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(ones + 512);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.y * UN_CH, co0 = blockIdx.z * CO, splits = gridDim.x;
    const int tiles_x = (a.W + TC_TW - 1) / TC_TW, tiles_y = (a.H + TC_TH - 1) / TC_TH, ntiles = tiles_x * tiles_y * a.B;
    const bool first = c0 < a.c1, bias = c0 == 0;
    const __nv_bfloat16* src = first ? a.src1 : a.src2;
    const int cs = first ? a.c1s : a.c2s, mode = first ? a.mode1 : a.mode2, cb = first ? c0 : c0 - a.c1;
    if (__syncthreads_or(*(volatile int*)status)) return;  // an earlier CTA's wait ran out: nothing is allocated yet
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(DW_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(smem_u32(mbar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    if (tid < 128) reinterpret_cast<uint32_t*>(ones)[tid] = 0x3F803F80u;  // bf16 ones, 16 columns x 16 pixels
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tslot;
    constexpr uint32_t MN = (1u << 15) | (1u << 16);  // A and B MN-major
    constexpr uint32_t IDESC = umma_idesc_bf16(96) | MN, IDESC1 = umma_idesc_bf16(16) | MN;

    uint4 xr[XQ], zr[ZQ];
    auto fetch = [&](int tile) {
        const int b = tile / (tiles_x * tiles_y), tr = tile % (tiles_x * tiles_y);
        const int x0 = (tr % tiles_x) * TC_TW, y0 = (tr / tiles_x) * TC_TH;
#pragma unroll
        for (int q = 0; q < ZQ; q++) {
            const int i = tid + q * DW_THREADS, pix = i / ZV, v = i % ZV, yy = y0 + pix / TC_TW, xx = x0 + pix % TC_TW;
            zr[q] = make_uint4(0u, 0u, 0u, 0u);
            if (yy < a.H && xx < a.W)
                zr[q] = *reinterpret_cast<const uint4*>(dz + (((size_t)b * a.H + yy) * a.W + xx) * a.cout + co0 + 8 * v);
        }
#pragma unroll
        for (int q = 0; q < XQ; q++) {
            const int i = tid + q * DW_THREADS, pix = i >> 2, v = i & 3, yy = y0 - 1 + pix / TC_WP, xx = x0 - 1 + pix % TC_WP;
            xr[q] = make_uint4(0u, 0u, 0u, 0u);
            if (i < XU && yy >= 0 && yy < a.H && xx >= 0 && xx < a.W) xr[q] = load8(src, cs, mode, b, yy, xx, a.H, a.W, cb + 8 * v);
        }
    };
    // a warp's sums: its lane quarter's couts, every other 16 of the 288 columns (the quarter's other warp has the rest)
    const bool reads = 32 * (warp & 3) < CO;
    const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    float sum[DW_BLOCKS][16], dbs = 0.f;
#pragma unroll
    for (int h = 0; h < DW_BLOCKS; h++)
#pragma unroll
        for (int q = 0; q < 16; q++) sum[h][q] = 0.f;
    // tile n's MMAs are done: its sums out of the TMEM, before the next tile's take their place
    auto take = [&](int n) {
        if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(mbar), (uint32_t)(n & 1)))) return false;
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (reads) {
#pragma unroll
            for (int h = 0; h < DW_BLOCKS; h++) {
                uint32_t r[16];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                      "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                    : "r"(tq + (uint32_t)((2 * h + (warp >> 2)) * 16)));
                asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
                for (int q = 0; q < 16; q++) sum[h][q] += __uint_as_float(r[q]);
            }
            if (bias && warp < 4) {
                uint32_t r;
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(tq + DW_DB_COL));
                asm volatile("tcgen05.wait::ld.sync.aligned;");
                dbs += __uint_as_float(r);
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        return true;
    };
    bool ok = true;
    int it = 0;
    fetch(blockIdx.x);
    for (int tile = blockIdx.x; tile < ntiles; tile += splits, it++) {
        // two stages in turn: the MMAs of two tiles ago, which read this one, were done before those of the last tile began
        unsigned char* Z = dw_smem + (it & 1) * STAGE;
        unsigned char* X = Z + ZV * ZP;
#pragma unroll
        for (int q = 0; q < ZQ; q++) {
            const int i = tid + q * DW_THREADS, pix = i / ZV, v = i % ZV;
            *reinterpret_cast<uint4*>(Z + v * ZP + pix * 16) = zr[q];
        }
#pragma unroll
        for (int q = 0; q < XQ; q++) {
            const int i = tid + q * DW_THREADS, pix = i >> 2, v = i & 3, r = pix / TC_WP, c = pix % TC_WP;
            if (i >= XU) break;
#pragma unroll
            for (int kx = 0; kx < 3; kx++)
                if (c >= kx && c < kx + TC_TW) *reinterpret_cast<uint4*>(X + (kx * 4 + v) * DW_XPLANE + (r * TC_TW + c - kx) * 16) = xr[q];
        }
        if (tile + splits < ntiles) fetch(tile + splits);  // in flight across the barrier and the MMAs
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (it > 0) ok = take(it - 1);
        if (!__syncthreads_and(ok)) {
            ok = false;
            break;
        }
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t zb = smem_u32(Z), xb = smem_u32(X);
#pragma unroll 1
            for (int j = 0; j < 8; j++) {  // 16 pixels (two tile rows) per K-step
                const uint64_t da = umma_desc(zb + j * 256, 128, ZP);
                const uint32_t acc = j > 0 ? 1u : 0u;
#pragma unroll
                for (int ky = 0; ky < 3; ky++) umma_bf16(tmem + ky * 96, da, umma_desc(xb + (2 * j + ky) * 128, 128, DW_XPLANE), IDESC, acc);
                if (bias) umma_bf16(tmem + DW_DB_COL, da, umma_desc(smem_u32(ones), 128, 256), IDESC1, acc);
            }
            umma_commit(smem_u32(mbar));
        }
    }
    if (ok) ok = take(it - 1);
    ok = __syncthreads_and(ok) != 0;
    if (!ok) {
        // a wait ran out: flag it, give the MMAs in flight a second bounded wait, free the TMEM, return
        if (tid == 0) atomicOr(status, 0x200);
        mbar_wait(smem_u32(mbar), (uint32_t)((it - 1) & 1));
    } else if (reads) {
        const int m = 32 * (warp & 3) + lane;  // this lane's cout
#pragma unroll
        for (int h = 0; h < DW_BLOCKS; h++) {
            const int col = (2 * h + (warp >> 2)) * 16;
            float* o = dw + ((size_t)(col / 32) * a.cout + co0 + m) * a.cin + c0 + col % 32;
#pragma unroll
            for (int q = 0; q < 16; q += 4) red_add4(o + q, sum[h][q], sum[h][q + 1], sum[h][q + 2], sum[h][q + 3]);
        }
        if (bias && warp < 4) atomicAdd(&db[co0 + m], dbs);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(DW_COLS));
}

// Adam on the FP32 masters, then the bf16 forward copy and the flipped,
// transposed copy the dX conv reads: wt[8 - tap][ci][co] = w[tap][co][ci].
__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ gw, float* __restrict__ m, float* __restrict__ v, size_t n,
                            float lr, float b1, float b2, float c1, float c2, float eps, const unsigned char* __restrict__ mask) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (mask && !mask[i]) continue;
        const float gr = gw[i];
        const float mi = b1 * m[i] + (1.f - b1) * gr, vi = b2 * v[i] + (1.f - b2) * gr * gr;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}
// The tcgen05 path's packing of a [tap][n][c] weight: [n / N][c / 32][tap][c % 32 / 8][n % N][c % 8], N = tc_block(nn).
__device__ __forceinline__ size_t pack_at(int tap, int n, int c, int nn, int cc) {
    const int N = tc_block(nn);
    return ((((size_t)(n / N) * (cc / 32) + c / 32) * 9 + tap) * 4 + c % 32 / 8) * N * 8 + (size_t)(n % N) * 8 + c % 8;
}
// wb = w, wt its flipped transpose for dX, and both packed (wp, wtp)
__global__ void cast_weights_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ wb, __nv_bfloat16* __restrict__ wt,
                                    __nv_bfloat16* __restrict__ wp, __nv_bfloat16* __restrict__ wtp, int cout, int cin) {
    const size_t n = (size_t)9 * cout * cin;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int ci = (int)(i % cin), co = (int)((i / cin) % cout), tap = (int)(i / ((size_t)cin * cout));
        const __nv_bfloat16 v = __float2bfloat16_rn(w[i]);
        wb[i] = v;
        wt[((size_t)(8 - tap) * cin + ci) * cout + co] = v;
        wp[pack_at(tap, co, ci, cout, cin)] = v;
        wtp[pack_at(8 - tap, ci, co, cin, cout)] = v;
    }
}

// ------------------------------------------------------------ input / output
// The network's input from the depth grid's planes (dw x dh): 2x2 means
// (clamped at the edge) onto a grid padded to a multiple of 8, channels
// (guide, d / dmax, conf), the rest zero; d_in keeps d / dmax in f32.
__global__ void unet_input_kernel(const float* __restrict__ guide, const float* __restrict__ d, const float* __restrict__ conf, int dw,
                                  int dh, float inv_dmax, int H, int W, int b, __nv_bfloat16* __restrict__ in, float* __restrict__ d_in) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    float s[3] = {0.f, 0.f, 0.f};
    for (int dy = 0; dy < 2; dy++)
        for (int dx = 0; dx < 2; dx++) {
            const int sx = min(2 * x + dx, dw - 1), sy = min(2 * y + dy, dh - 1);
            const size_t k = (size_t)sy * dw + sx;
            s[0] += guide[k];
            s[1] += d[k] * inv_dmax;
            s[2] += conf[k];
        }
    const size_t p = ((size_t)b * H + y) * W + x;
    // the pixel's 32 channels, 3 live, as four 16-byte stores (channel by channel: 49 us on 512 x 384, 6 here)
    uint4* o = reinterpret_cast<uint4*>(in + p * UN_CH);
    const uint32_t c01 = bf2_as_u32(__floats2bfloat162_rn(0.25f * s[0], 0.25f * s[1]));
    const uint32_t c23 = bf2_as_u32(__floats2bfloat162_rn(fminf(0.25f * s[2], 4.f), 0.f));
    o[0] = make_uint4(c01, c23, 0u, 0u);
    for (int q = 1; q < UN_CH / 8; q++) o[q] = make_uint4(0u, 0u, 0u, 0u);
    d_in[p] = 0.25f * s[1];
}
// y = d_in + out0 on the network grid; bilinear back to the depth grid, times dmax
__global__ void unet_output_kernel(const float* __restrict__ d_in, const float* __restrict__ out0, int H, int W, int b, int dw, int dh,
                                   float dmax, float* __restrict__ x0) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= dw || y >= dh) return;
    const float fx = fminf(fmaxf((x + 0.5f) * 0.5f - 0.5f, 0.f), (float)(W - 1));
    const float fy = fminf(fmaxf((y + 0.5f) * 0.5f - 0.5f, 0.f), (float)(H - 1));
    const int xa = (int)fx, ya = (int)fy, xb = min(xa + 1, W - 1), yb = min(ya + 1, H - 1);
    const float tx = fx - xa, ty = fy - ya;
    const size_t base = (size_t)b * H * W;
    auto Y = [&](int yy, int xx) { const size_t k = base + (size_t)yy * W + xx; return d_in[k] + out0[k]; };
    const float v = (1.f - ty) * ((1.f - tx) * Y(ya, xa) + tx * Y(ya, xb)) + ty * ((1.f - tx) * Y(yb, xa) + tx * Y(yb, xb));
    x0[(size_t)y * dw + x] = fminf(fmaxf(v, 0.f), 1.f) * dmax;
}
// MSE on the network grid: loss partials and dL/dout0 = 2 (d_in + out0 - t) / n
__global__ void mse_kernel(const float* __restrict__ d_in, const float* __restrict__ out0, const float* __restrict__ tgt, size_t n,
                           float* __restrict__ dout0, double* __restrict__ loss) {
    double s = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float e = d_in[i] + out0[i] - tgt[i];
        dout0[i] = 2.f * e / (float)n;
        s += (double)e * e;
    }
    __shared__ double red[256];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, red[0] / (double)n);
}

// ------------------------------------------------------------------- network
struct Layer {
    int src1, mode1, c1, src2, mode2, c2, cout, level, relu;
    size_t woff, boff;  // offsets in the parameter arrays
};
// tensor t (0 = input, i + 1 = output of layer i): level, channels
static const int N_LAYERS = 15;
static std::vector<Layer> unet_layers() {
    std::vector<Layer> L;
    auto add = [&](int s1, int m1, int c1, int s2, int m2, int c2, int co, int lv, int relu) {
        L.push_back(Layer{s1, m1, c1, s2, m2, c2, co, lv, relu, 0, 0});
    };
    add(0, SRC_SAME, 32, -1, 0, 0, 32, 0, 1);      // 0  E0a  (input: 3 channels of 32)
    add(1, SRC_SAME, 32, -1, 0, 0, 32, 0, 1);      // 1  E0b  skip0
    add(2, SRC_POOL, 32, -1, 0, 0, 64, 1, 1);      // 2  E1a
    add(3, SRC_SAME, 64, -1, 0, 0, 64, 1, 1);      // 3  E1b  skip1
    add(4, SRC_POOL, 64, -1, 0, 0, 128, 2, 1);     // 4  E2a
    add(5, SRC_SAME, 128, -1, 0, 0, 128, 2, 1);    // 5  E2b  skip2
    add(6, SRC_POOL, 128, -1, 0, 0, 256, 3, 1);    // 6  B3a
    add(7, SRC_SAME, 256, -1, 0, 0, 256, 3, 1);    // 7  B3b
    add(8, SRC_UP, 256, 6, SRC_SAME, 128, 128, 2, 1);  // 8  D2a = up(B3b) ++ skip2
    add(9, SRC_SAME, 128, -1, 0, 0, 128, 2, 1);    // 9  D2b
    add(10, SRC_UP, 128, 4, SRC_SAME, 64, 64, 1, 1);   // 10 D1a = up(D2b) ++ skip1
    add(11, SRC_SAME, 64, -1, 0, 0, 64, 1, 1);     // 11 D1b
    add(12, SRC_UP, 64, 2, SRC_SAME, 32, 32, 0, 1);    // 12 D0a = up(D1b) ++ skip0
    add(13, SRC_SAME, 32, -1, 0, 0, 32, 0, 1);     // 13 D0b
    add(14, SRC_SAME, 32, -1, 0, 0, 32, 0, 0);     // 14 OUT  (channel 0 only; linear)
    size_t wo = 0, bo = 0;
    for (auto& l : L) {
        l.woff = wo;
        l.boff = bo;
        wo += (size_t)9 * l.cout * (l.c1 + l.c2);
        bo += l.cout;
    }
    return L;
}

}  // namespace lsb

using namespace lsb;

struct lsb_unet {
    int device = 0;
    cudaStream_t s = nullptr;
    std::vector<Layer> layers;
    size_t nw = 0, nb = 0;  // parameter counts
    // FP32 masters, grads, Adam moments (weights then biases, one array each)
    float *w = nullptr, *gw = nullptr, *mw = nullptr, *vw = nullptr;
    float *b = nullptr, *gb = nullptr, *mb = nullptr, *vb = nullptr;
    unsigned char* wmask = nullptr;  // trainable weights (the output layer keeps channels 1.. at zero)
    unsigned char* bmask = nullptr;
    __nv_bfloat16 *wb = nullptr, *wt = nullptr, *wp = nullptr, *wtp = nullptr;
    int step = 0;
    // activations for the current shape
    int B = 0, H = 0, W = 0;
    std::vector<__nv_bfloat16*> act;  // bf16 [B][h_l][w_l][c]
    std::vector<float*> dx;           // training: each layer's dX (f32, its grid, its input channels), read by its sources' dZ
    float *out0 = nullptr, *dout0 = nullptr, *d_in = nullptr, *x0 = nullptr;
    __nv_bfloat16* dz = nullptr;
    double* loss = nullptr;
    double* loss_host = nullptr;
    std::vector<void*> shape_allocs;
    int* status = nullptr;  // device error word of the tcgen05 convolution (a bounded wait ran out)
    bool tc = true;         // the 3x3 convolutions on tcgen05 (false: mma.sync, for comparison)
    cudaEvent_t fev[2] = {nullptr, nullptr};  // around the last forward pass's layers on s
    float fwd_ms = 0.f;
};

static char* un_err(const std::string& s) {
    char* p = (char*)malloc(s.size() + 1);
    memcpy(p, s.c_str(), s.size() + 1);
    return p;
}
#define UTRY(x)                                                                                 \
    do {                                                                                        \
        cudaError_t _e = (x);                                                                   \
        if (_e != cudaSuccess) return un_err(std::string("unet: ") + cudaGetErrorString(_e)); \
    } while (0)

static int ugrid(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 148 * 8); }

static size_t act_channels(const lsb_unet* u, int t) { return t == 0 ? 32 : u->layers[t - 1].cout; }
static int act_level(const lsb_unet* u, int t) { return t == 0 ? 0 : u->layers[t - 1].level; }

static void free_shape(lsb_unet* u) {
    for (void* p : u->shape_allocs) cudaFree(p);
    u->shape_allocs.clear();
    u->act.clear();
    u->dx.clear();
    u->B = u->H = u->W = 0;
}

static cudaError_t ensure_shape(lsb_unet* u, int B, int H, int W, bool train) {
    if (u->B == B && u->H == H && u->W == W && (!train || !u->dx.empty())) return cudaSuccess;
    free_shape(u);
    auto get = [&](size_t bytes, void** p) {
        cudaError_t e = lsb_dev_alloc(p, std::max<size_t>(bytes, 16));
        if (e == cudaSuccess) u->shape_allocs.push_back(*p);
        return e;
    };
    size_t maxc = 0;
    for (int t = 0; t <= N_LAYERS; t++) {
        const int lv = act_level(u, t);
        const size_t px = (size_t)B * (H >> lv) * (W >> lv), c = act_channels(u, t);
        void* p;
        cudaError_t e = get(px * c * sizeof(__nv_bfloat16), &p);
        if (e != cudaSuccess) return e;
        u->act.push_back((__nv_bfloat16*)p);
        maxc = std::max(maxc, px * c);
    }
    for (size_t i = 0; i < u->layers.size() && train; i++) {
        const Layer& l = u->layers[i];
        void* p = nullptr;
        cudaError_t e = i == 0 ? cudaSuccess : get((size_t)B * (H >> l.level) * (W >> l.level) * (l.c1 + l.c2) * sizeof(float), &p);
        if (e != cudaSuccess) {
            u->dx.clear();
            return e;
        }
        u->dx.push_back((float*)p);
    }
    const size_t px0 = (size_t)B * H * W;
    void* p;
    cudaError_t e;
    if ((e = get(px0 * sizeof(float), &p)) != cudaSuccess) return e;
    u->out0 = (float*)p;
    if ((e = get(px0 * sizeof(float), &p)) != cudaSuccess) return e;
    u->d_in = (float*)p;
    if (train) {
        if ((e = get(px0 * sizeof(float), &p)) != cudaSuccess) return e;
        u->dout0 = (float*)p;
        if ((e = get(maxc * sizeof(__nv_bfloat16), &p)) != cudaSuccess) return e;
        u->dz = (__nv_bfloat16*)p;
    }
    u->B = B;
    u->H = H;
    u->W = W;
    return cudaSuccess;
}

template <int N>
static cudaError_t conv_tc_launch(const ConvArgs& a, int* status, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(conv3x3_tc_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc_smem(N));
    if (e != cudaSuccess) return e;
    const int ntiles = ((a.W + TC_TW - 1) / TC_TW) * ((a.H + TC_TH - 1) / TC_TH) * a.B, nblk = a.cout / N;
    const dim3 grid(std::min(ntiles, std::max(1, 148 / nblk)), nblk);
    // the layer before releases this one's CTAs early (griddepcontrol): each sets up as soon as its SM is free
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = tc_smem(N);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    lsb_launched();
    return cudaLaunchKernelEx(&cfg, conv3x3_tc_kernel<N>, a, status);
}

static cudaError_t conv_launch(const ConvArgs& a, cudaStream_t s, int* status = nullptr, bool tc = false) {
    // tcgen05: every layer's cin is a multiple of 32 and its cout a multiple of one of the kernel's N
    if (tc && status && a.wp && a.cin % UN_CH == 0) {
        switch (tc_block(a.cout)) {
            case 32: return conv_tc_launch<32>(a, status, s);
            case 64: return conv_tc_launch<64>(a, status, s);
            case 96: return conv_tc_launch<96>(a, status, s);
            case 128: return conv_tc_launch<128>(a, status, s);
            default: break;
        }
    }
    const int NT = a.cout % 64 == 0 ? 64 : 32;
    const size_t smem = (size_t)(UN_HP * UN_WP + 9 * NT) * UN_LD * sizeof(__nv_bfloat16);
    const dim3 grid(((a.W + UN_TW - 1) / UN_TW) * ((a.H + UN_TH - 1) / UN_TH), a.cout / NT, a.B);
    if (NT == 64) {
        cudaFuncSetAttribute(conv3x3_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        lsb_launched(), conv3x3_kernel<64><<<grid, UN_THREADS, smem, s>>>(a);
    } else {
        cudaFuncSetAttribute(conv3x3_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        lsb_launched(), conv3x3_kernel<32><<<grid, UN_THREADS, smem, s>>>(a);
    }
    return cudaGetLastError();
}

template <int CO>
static cudaError_t dw_launch_co(const ConvArgs& a, const __nv_bfloat16* dz, float* dw, float* db, int* status, cudaStream_t s) {
    const size_t smem = dw_smem_bytes(CO);
    cudaError_t e = cudaFuncSetAttribute(conv_dw_kernel<CO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int ntiles = ((a.W + TC_TW - 1) / TC_TW) * ((a.H + TC_TH - 1) / TC_TH) * a.B;
    const int blocks = (a.cin / UN_CH) * (a.cout / CO);
    // one CTA per SM (a CTA takes all of the TMEM): the tiles split so that the channel blocks fill the 148 SMs
    const dim3 grid(std::max(1, std::min(ntiles, 148 / blocks)), a.cin / UN_CH, a.cout / CO);
    lsb_launched(), conv_dw_kernel<CO><<<grid, DW_THREADS, smem, s>>>(a, dz, dw, db, status);
    return cudaGetLastError();
}
static cudaError_t dw_launch(const ConvArgs& a, const __nv_bfloat16* dz, float* dw, float* db, int* status, cudaStream_t s) {
    if (a.cout % 128 == 0) return dw_launch_co<128>(a, dz, dw, db, status, s);
    return a.cout == 64 ? dw_launch_co<64>(a, dz, dw, db, status, s) : dw_launch_co<32>(a, dz, dw, db, status, s);
}

static ConvArgs layer_args(const lsb_unet* u, int i) {
    const Layer& l = u->layers[i];
    ConvArgs a{};
    a.src1 = u->act[l.src1];
    a.c1 = l.c1;
    a.c1s = (int)act_channels(u, l.src1);
    a.mode1 = l.mode1;
    a.src2 = l.src2 >= 0 ? u->act[l.src2] : nullptr;
    a.c2s = l.src2 >= 0 ? (int)act_channels(u, l.src2) : 0;
    a.mode2 = l.mode2;
    a.cin = l.c1 + l.c2;
    a.cout = l.cout;
    a.w = u->wb + l.woff;
    a.wp = u->wp + l.woff;
    a.bias = u->b + l.boff;
    a.relu = l.relu;
    a.B = u->B;
    a.H = u->H >> l.level;
    a.W = u->W >> l.level;
    return a;
}

static cudaError_t unet_forward(lsb_unet* u) {
    for (int i = 0; i < N_LAYERS; i++) {
        ConvArgs a = layer_args(u, i);
        const bool last = i == N_LAYERS - 1;
        a.out = u->act[i + 1];
        a.out_c0 = last ? u->out0 : nullptr;
        cudaError_t e = conv_launch(a, u->s, u->status, u->tc);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

static cudaError_t cast_all(lsb_unet* u) {
    for (auto& l : u->layers) {
        lsb_launched(), cast_weights_kernel<<<ugrid((size_t)9 * l.cout * (l.c1 + l.c2)), 256, 0, u->s>>>(u->w + l.woff, u->wb + l.woff, u->wt + l.woff,
                                                                                                      u->wp + l.woff, u->wtp + l.woff, l.cout,
                                                                                                      l.c1 + l.c2);
    }
    return cudaGetLastError();
}

extern "C" char* lsb_unet_create(int32_t device, uint64_t seed, lsb_unet** out) {
    *out = nullptr;
    lsb_unet* u = new lsb_unet();
    u->device = device;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        delete u;
        return un_err(std::string("unet: ") + cudaGetErrorString(e));
    }
    u->layers = unet_layers();
    for (auto& l : u->layers) {
        u->nw = l.woff + (size_t)9 * l.cout * (l.c1 + l.c2);
        u->nb = l.boff + l.cout;
    }
    std::vector<float> w(u->nw, 0.f), b(u->nb, 0.f);
    std::vector<unsigned char> wm(u->nw, 1), bm(u->nb, 1);
    std::mt19937_64 rng(seed);
    std::normal_distribution<float> nd(0.f, 1.f);
    for (size_t li = 0; li < u->layers.size(); li++) {
        const Layer& l = u->layers[li];
        const int cin = l.c1 + l.c2;
        const int fan_in = 9 * (li == 0 ? 3 : cin);
        const float sd = li + 1 == u->layers.size() ? 1e-3f : std::sqrt(2.f / fan_in);
        for (int tap = 0; tap < 9; tap++)
            for (int co = 0; co < l.cout; co++)
                for (int ci = 0; ci < cin; ci++) {
                    const size_t k = l.woff + ((size_t)tap * l.cout + co) * cin + ci;
                    const bool live = (li != 0 || ci < 3) && (li + 1 != u->layers.size() || co == 0);
                    w[k] = live ? sd * nd(rng) : 0.f;
                    wm[k] = live;
                }
        for (int co = 0; co < l.cout; co++) bm[l.boff + co] = li + 1 != u->layers.size() || co == 0;
    }
    auto alloc = [&](void** p, size_t bytes) -> bool {
        if (lsb_dev_alloc(p, bytes) != cudaSuccess) return false;
        return cudaMemset(*p, 0, bytes) == cudaSuccess;
    };
    bool ok = alloc((void**)&u->w, u->nw * 4) && alloc((void**)&u->gw, u->nw * 4) && alloc((void**)&u->mw, u->nw * 4) &&
              alloc((void**)&u->vw, u->nw * 4) && alloc((void**)&u->b, u->nb * 4) && alloc((void**)&u->gb, u->nb * 4) &&
              alloc((void**)&u->mb, u->nb * 4) && alloc((void**)&u->vb, u->nb * 4) && alloc((void**)&u->wmask, u->nw) &&
              alloc((void**)&u->bmask, u->nb) && alloc((void**)&u->wb, u->nw * 2) && alloc((void**)&u->wt, u->nw * 2) &&
              alloc((void**)&u->wp, u->nw * 2) && alloc((void**)&u->wtp, u->nw * 2) &&
              alloc((void**)&u->loss, 8) && alloc((void**)&u->status, 4) &&
              cudaHostAlloc((void**)&u->loss_host, 8, cudaHostAllocDefault) == cudaSuccess &&
              cudaStreamCreateWithFlags(&u->s, cudaStreamNonBlocking) == cudaSuccess;
    if (!ok) {
        lsb_unet_destroy(u);
        return un_err("unet: device allocation failed");
    }
    cudaMemcpy(u->w, w.data(), u->nw * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(u->b, b.data(), u->nb * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(u->wmask, wm.data(), u->nw, cudaMemcpyHostToDevice);
    cudaMemcpy(u->bmask, bm.data(), u->nb, cudaMemcpyHostToDevice);
    e = cast_all(u);
    if (e == cudaSuccess) e = cudaStreamSynchronize(u->s);
    if (e != cudaSuccess) {
        lsb_unet_destroy(u);
        return un_err(std::string("unet: ") + cudaGetErrorString(e));
    }
    *out = u;
    return nullptr;
}

extern "C" void lsb_unet_destroy(lsb_unet* u) {
    if (!u) return;
    if (u->s) cudaStreamSynchronize(u->s);
    free_shape(u);
    for (void* p : {(void*)u->w, (void*)u->gw, (void*)u->mw, (void*)u->vw, (void*)u->b, (void*)u->gb, (void*)u->mb, (void*)u->vb,
                    (void*)u->wmask, (void*)u->bmask, (void*)u->wb, (void*)u->wt, (void*)u->wp, (void*)u->wtp, (void*)u->loss, (void*)u->status})
        if (p) cudaFree(p);
    if (u->loss_host) cudaFreeHost(u->loss_host);
    for (cudaEvent_t v : u->fev)
        if (v) cudaEventDestroy(v);
    if (u->s) cudaStreamDestroy(u->s);
    delete u;
}

// The device error word: a tcgen05 convolution whose bounded wait ran out (its output is not written).
static char* conv_status(lsb_unet* u) {
    int st = 0;
    UTRY(cudaMemcpy(&st, u->status, sizeof st, cudaMemcpyDeviceToHost));
    if (st) {
        cudaMemset(u->status, 0, sizeof st);
        return un_err("unet: a tensor-core convolution's wait for its MMAs ran out");
    }
    return nullptr;
}

extern "C" char* lsb_unet_set_conv(lsb_unet* u, uint32_t path) {
    if (!u) return un_err("unet: null network");
    if (path > 1) return un_err("unet: conv path must be 0 (tcgen05) or 1 (mma.sync)");
    u->tc = path == 0;
    return nullptr;
}

extern "C" void lsb_unet_sizes(const lsb_unet* u, uint64_t* n_weights, uint64_t* n_biases) {
    *n_weights = u->nw;
    *n_biases = u->nb;
}

extern "C" char* lsb_unet_get_params(lsb_unet* u, float* w, float* b, float* gw, float* gb) {
    UTRY(cudaStreamSynchronize(u->s));
    if (w) UTRY(cudaMemcpy(w, u->w, u->nw * 4, cudaMemcpyDeviceToHost));
    if (b) UTRY(cudaMemcpy(b, u->b, u->nb * 4, cudaMemcpyDeviceToHost));
    if (gw) UTRY(cudaMemcpy(gw, u->gw, u->nw * 4, cudaMemcpyDeviceToHost));
    if (gb) UTRY(cudaMemcpy(gb, u->gb, u->nb * 4, cudaMemcpyDeviceToHost));
    return nullptr;
}

extern "C" char* lsb_unet_set_params(lsb_unet* u, const float* w, const float* b) {
    UTRY(cudaStreamSynchronize(u->s));
    UTRY(cudaMemcpy(u->w, w, u->nw * 4, cudaMemcpyHostToDevice));
    UTRY(cudaMemcpy(u->b, b, u->nb * 4, cudaMemcpyHostToDevice));
    UTRY(cast_all(u));
    UTRY(cudaStreamSynchronize(u->s));
    return nullptr;
}

// in: device [B][H][W][32] bf16 (lsb_unet_prepare's layout), d_in: device [B][H][W] f32
static char* stage_batch(lsb_unet* u, const void* in, const float* d_in, int B, int H, int W, bool train) {
    if (H % 8 || W % 8 || H < 8 || W < 8) return un_err("unet: the grid must be a multiple of 8 on both sides");
    UTRY(ensure_shape(u, B, H, W, train));
    UTRY(cudaMemcpyAsync(u->act[0], in, (size_t)B * H * W * UN_CH * 2, cudaMemcpyDeviceToDevice, u->s));
    UTRY(cudaMemcpyAsync(u->d_in, d_in, (size_t)B * H * W * 4, cudaMemcpyDeviceToDevice, u->s));
    return nullptr;
}

extern "C" char* lsb_unet_forward(lsb_unet* u, const void* in_dev, const float* d_in_dev, uint32_t B, uint32_t H, uint32_t W,
                                  float* out0_dev) {
    if (char* er = stage_batch(u, in_dev, d_in_dev, (int)B, (int)H, (int)W, false)) return er;
    for (cudaEvent_t& v : u->fev)
        if (!v) UTRY(cudaEventCreate(&v));
    UTRY(cudaEventRecord(u->fev[0], u->s));
    UTRY(unet_forward(u));
    UTRY(cudaEventRecord(u->fev[1], u->s));
    if (out0_dev) UTRY(cudaMemcpyAsync(out0_dev, u->out0, (size_t)B * H * W * 4, cudaMemcpyDeviceToDevice, u->s));
    UTRY(cudaStreamSynchronize(u->s));
    UTRY(cudaEventElapsedTime(&u->fwd_ms, u->fev[0], u->fev[1]));
    return conv_status(u);
}

extern "C" char* lsb_unet_forward_ms(lsb_unet* u, float* ms) {
    if (!u || !ms) return un_err("unet: null argument");
    *ms = u->fwd_ms;
    return nullptr;
}

static cudaError_t unet_backward(lsb_unet* u) {
    cudaMemsetAsync(u->gw, 0, u->nw * 4, u->s);
    cudaMemsetAsync(u->gb, 0, u->nb * 4, u->s);
    for (int i = N_LAYERS - 1; i >= 0; i--) {
        const Layer& l = u->layers[i];
        ConvArgs a = layer_args(u, i);
        const size_t npx = (size_t)a.B * a.H * a.W;
        if (i == N_LAYERS - 1)
            lsb_launched(), out_grad_kernel<<<ugrid(npx * 4), 256, 0, u->s>>>(u->dout0, u->dz, npx);
        else {
            GradUse use[2] = {};
            int uses = 0;
            for (int j = N_LAYERS - 1; j > i; j--) {  // in the order their dX exist: the last layer's first
                const Layer& q = u->layers[j];
                const int in = q.src1 == i + 1 ? 0 : q.src2 == i + 1 ? q.c1 : -1;
                if (in >= 0) use[uses++] = GradUse{u->dx[j], q.c1 + q.c2, in, in ? q.mode2 : q.mode1, u->H >> q.level, u->W >> q.level};
            }
            const size_t items = npx * l.cout / 8;
            lsb_launched(), grad_gather_kernel<<<ugrid(items), 256, 0, u->s>>>(use[0], use[1], uses, u->act[i + 1], u->dz, a.H, a.W, l.cout, items,
                                                                               l.relu);
        }
        const int cin = l.c1 + l.c2;
        cudaError_t e = dw_launch(a, u->dz, u->gw + l.woff, u->gb + l.boff, u->status, u->s);
        if (e != cudaSuccess) return e;
        if (i == 0) continue;  // no gradient for the input
        ConvArgs d{};
        d.src1 = u->dz;
        d.c1 = l.cout;
        d.c1s = l.cout;
        d.mode1 = SRC_SAME;
        d.cin = l.cout;
        d.cout = cin;
        d.w = u->wt + l.woff;
        d.wp = u->wtp + l.woff;
        d.out_f32 = u->dx[i];
        d.B = a.B;
        d.H = a.H;
        d.W = a.W;
        e = conv_launch(d, u->s, u->status, u->tc);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

// One step on a batch: forward, MSE against target (d / dmax on the network
// grid), backward; Adam when lr > 0. loss_out gets the batch's MSE.
extern "C" char* lsb_unet_train_step(lsb_unet* u, const void* in_dev, const float* d_in_dev, const float* target_dev, uint32_t B,
                                     uint32_t H, uint32_t W, float lr, double* loss_out) {
    if (char* er = stage_batch(u, in_dev, d_in_dev, (int)B, (int)H, (int)W, true)) return er;
    UTRY(unet_forward(u));
    const size_t n = (size_t)B * H * W;
    UTRY(cudaMemsetAsync(u->loss, 0, 8, u->s));
    lsb_launched(), mse_kernel<<<ugrid(n), 256, 0, u->s>>>(u->d_in, u->out0, target_dev, n, u->dout0, u->loss);
    UTRY(unet_backward(u));
    if (lr > 0.f) {
        u->step++;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.f - std::pow(b1, (float)u->step), c2 = 1.f - std::pow(b2, (float)u->step);
        lsb_launched(), adam_kernel<<<ugrid(u->nw), 256, 0, u->s>>>(u->w, u->gw, u->mw, u->vw, u->nw, lr, b1, b2, c1, c2, 1e-8f, u->wmask);
        lsb_launched(), adam_kernel<<<ugrid(u->nb), 256, 0, u->s>>>(u->b, u->gb, u->mb, u->vb, u->nb, lr, b1, b2, c1, c2, 1e-8f, u->bmask);
        UTRY(cast_all(u));
    }
    UTRY(cudaMemcpyAsync(u->loss_host, u->loss, 8, cudaMemcpyDeviceToHost, u->s));
    UTRY(cudaStreamSynchronize(u->s));
    if (loss_out) *loss_out = *u->loss_host;
    return conv_status(u);
}

// The network input of one depth grid (device planes dw x dh): in [H][W][32]
// bf16 and d_in [H][W] f32 at batch index b, H = round_up(ceil(dh/2), 8), W likewise.
extern "C" void lsb_unet_grid(uint32_t dw, uint32_t dh, uint32_t* H, uint32_t* W) {
    *W = ((dw + 1) / 2 + 7) / 8 * 8;
    *H = ((dh + 1) / 2 + 7) / 8 * 8;
}
extern "C" char* lsb_unet_prepare(const float* guide, const float* d, const float* conf, uint32_t dw, uint32_t dh, float dmax,
                                  void* in_dev, float* d_in_dev, uint32_t b, void* stream) {
    uint32_t H, W;
    lsb_unet_grid(dw, dh, &H, &W);
    const dim3 blk(32, 8), grd((W + 31) / 32, (H + 7) / 8);
    lsb_launched(), unet_input_kernel<<<grd, blk, 0, (cudaStream_t)stream>>>(guide, d, conf, (int)dw, (int)dh, 1.f / std::max(dmax, 1e-6f),
                                                                             (int)H, (int)W, (int)b, (__nv_bfloat16*)in_dev, d_in_dev);
    UTRY(cudaGetLastError());
    return nullptr;
}

namespace lsb {
// The warm start for a depth grid: prepare, forward, back to the grid.
cudaError_t unet_warm_start(lsb_unet* u, const float* guide, const float* d, const float* conf, int dw, int dh, float dmax, float* x0,
                            cudaStream_t st) {
    uint32_t H, W;
    lsb_unet_grid((uint32_t)dw, (uint32_t)dh, &H, &W);
    cudaError_t e = ensure_shape(u, 1, (int)H, (int)W, false);
    if (e != cudaSuccess) return e;
    // the network runs on the caller's stream
    cudaStream_t keep = u->s;
    u->s = st;
    const dim3 blk(32, 8), grd((W + 31) / 32, (H + 7) / 8);
    lsb_launched(), unet_input_kernel<<<grd, blk, 0, st>>>(guide, d, conf, dw, dh, 1.f / std::max(dmax, 1e-6f), (int)H, (int)W, 0,
                                                           u->act[0], u->d_in);
    e = unet_forward(u);
    if (e == cudaSuccess) {
        const dim3 g2((dw + 31) / 32, (dh + 7) / 8);
        lsb_launched(), unet_output_kernel<<<g2, blk, 0, st>>>(u->d_in, u->out0, (int)H, (int)W, 0, dw, dh, dmax, x0);
        e = cudaGetLastError();
    }
    u->s = keep;
    return e;
}
}  // namespace lsb
