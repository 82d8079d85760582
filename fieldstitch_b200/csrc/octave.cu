// Float32 octave kernels: the tiled per-layer kernel (k_layer) and the fused layer groups (k_group).
//
// Reference: app/planesite/gsift.py:85-87 (separable mirror blur), 158-179 (layers, DoG,
// downsample), 244-267 (gradient magnitude / angle of gauss layers 1..3).
//
// Arithmetic is packed FP32x2 (__ffma2_rn / __fadd2_rn) with symmetric tap pairing
// w_0 x_0 + sum_j w_j (x_-j + x_j): a mirrored input gives a bit-identical mirrored output.
//
// Every plane (gauss layers, DoG, gradient, the next octave's base) has a row pitch P, the width
// rounded up to a multiple of four, so every row starts on a 16-byte boundary (32 for gradients)
// whatever the octave's width; the pad columns hold no data and may be written.
#include <cuda.h>

#include <cstring>

#include "fsb_internal.cuh"

namespace fsb {

__constant__ float2 c_tap2[6][14];   // (w_j, w_j) at distance j = 0..r of layer i's taps

int32_t upload_octave_taps(const float* taps, int stride, const int* counts) {
    float2 t[6][14] = {};
    for (int i = 0; i < 6; ++i) {
        const int r = counts[i] / 2;
        for (int j = 0; j <= r; ++j) t[i][j] = make_float2(taps[i * stride + r + j], taps[i * stride + r + j]);
    }
    FSB_CUDA(cudaMemcpyToSymbol(c_tap2, t, sizeof(t)));
    return FSB_OK;
}

namespace {

// radius of layer i's blur
__host__ __device__ constexpr int RAD(int i) { return i == 1 ? 5 : i == 2 ? 6 : i == 3 ? 8 : i == 4 ? 10 : i == 5 ? 13 : 0; }

// Four gradient pixels (magnitude, angle) to a 32-byte aligned address: one 32-byte store, so a lane
// fills whole sectors (two 16-byte stores 32 bytes apart per lane would send each sector twice).
__device__ __forceinline__ void st_grad4(float2* p, const float (&mg)[4], const float (&an)[4]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(mg[0]), "f"(an[0]), "f"(mg[1]),
                 "f"(an[1]), "f"(mg[2]), "f"(an[2]), "f"(mg[3]), "f"(an[3])
                 : "memory");
}
__device__ __forceinline__ int mir(int p, int n) {
    if (n == 1) return 0;
    while (p < 0 || p >= n) p = p < 0 ? -p : 2 * n - 2 - p;
    return p;
}

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }

// tap set TS held in registers for a whole pass (the empty asm keeps the compiler from re-reading
// the constant bank at every packed FMA, which takes no constant operand)
template <int TS, int r>
__device__ __forceinline__ void load_taps(float2 (&w)[r + 1]) {
#pragma unroll
    for (int j = 0; j <= r; ++j) {
        float2 t = c_tap2[TS][j];
        asm volatile("" : "+f"(t.x), "+f"(t.y));
        w[j] = t;
    }
}
// sum_j w_j x[r + j] over j = -r..r for two lanes at once, with symmetric pairing
// w_0 x_0 + sum_j w_j (x_-j + x_j); two accumulation chains (odd / even j) for latency hiding.
// The pair sums commute, so a mirrored window gives a bit-identical result.
template <int r>
__device__ __forceinline__ float2 blur_pairs_w(const float2* x, const float2 (&w)[r + 1]) {
    float2 a = __fmul2_rn(x[r], w[0]);
    float2 b = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = r; j >= 1; --j) {
        const float2 p = __fadd2_rn(x[r - j], x[r + j]);
        if (j & 1)
            b = __ffma2_rn(p, w[j], b);
        else
            a = __ffma2_rn(p, w[j], a);
    }
    return __fadd2_rn(a, b);
}

// Gradient magnitude and direction (degrees in [0, 360)) of four pixels for the default (float32)
// pyramid: magnitude by the approximate square root (within a few ulps of sqrt), direction by
// octant reduction to t = min/max in [0, 1] (approximate reciprocal) and an odd polynomial for
// atan(t) in degrees. The
// coefficients were fitted here by iteratively reweighted least squares on Chebyshev nodes (max
// error 2.2e-6 deg; 7.4e-6 deg with float32 evaluation), so the angle stays well inside the
// reference's 0.1 deg keypoint tolerance. atan2(0, 0) = 0 as in the reference (border pixels).
// Pixels go through in pairs with packed FP32x2 arithmetic; every multiply and add is explicitly
// rounded (nothing is contracted into a fused multiply-add), so each engine that calls this
// function computes the same bits.
// the hardware's approximate square root and reciprocal (a few ulps; sqrt of 0 is 0)
__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void fast_grad4(const float (&dx)[4], const float (&dy)[4], float (&mag)[4],
                                           float (&ang)[4]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float2 X = make_float2(dx[2 * h], dx[2 * h + 1]), Y = make_float2(dy[2 * h], dy[2 * h + 1]);
        const float2 d2 = __fadd2_rn(__fmul2_rn(X, X), __fmul2_rn(Y, Y));
        const float2 m = make_float2(sqrt_approx(d2.x), sqrt_approx(d2.y));
        const float ax0 = fabsf(X.x), ay0 = fabsf(Y.x), ax1 = fabsf(X.y), ay1 = fabsf(Y.y);
        const float mx0 = fmaxf(ax0, ay0), mn0 = fminf(ax0, ay0), mx1 = fmaxf(ax1, ay1), mn1 = fminf(ax1, ay1);
        // min / max with the maximum kept above zero: 0 / tiny = 0 where both components vanish
        const float2 t = __fmul2_rn(make_float2(mn0, mn1),
                                    make_float2(rcp_approx(fmaxf(mx0, 1e-30f)), rcp_approx(fmaxf(mx1, 1e-30f))));
        const float2 z = __fmul2_rn(t, t);
        float2 p = make_float2(-2.323089093e-01f, -2.323089093e-01f);
        p = __ffma2_rn(p, z, make_float2(1.252652928e+00f, 1.252652928e+00f));
        p = __ffma2_rn(p, z, make_float2(-3.203537344e+00f, -3.203537344e+00f));
        p = __ffma2_rn(p, z, make_float2(5.524570187e+00f, 5.524570187e+00f));
        p = __ffma2_rn(p, z, make_float2(-7.969057098e+00f, -7.969057098e+00f));
        p = __ffma2_rn(p, z, make_float2(1.142854019e+01f, 1.142854019e+01f));
        p = __ffma2_rn(p, z, make_float2(-1.909660354e+01f, -1.909660354e+01f));
        p = __ffma2_rn(p, z, make_float2(5.729574144e+01f, 5.729574144e+01f));
        float2 a = __fmul2_rn(p, t);   // atan(min/max) in degrees, [0, 45]
        float2 f = __fadd2_rn(make_float2(90.f, 90.f), make_float2(-a.x, -a.y));
        a = make_float2(ay0 > ax0 ? f.x : a.x, ay1 > ax1 ? f.y : a.y);
        f = __fadd2_rn(make_float2(180.f, 180.f), make_float2(-a.x, -a.y));
        a = make_float2(X.x < 0.f ? f.x : a.x, X.y < 0.f ? f.y : a.y);
        f = __fadd2_rn(make_float2(360.f, 360.f), make_float2(-a.x, -a.y));   // atan2 < 0 maps to a + 360
        a = make_float2(Y.x < 0.f ? f.x : a.x, Y.y < 0.f ? f.y : a.y);
        mag[2 * h] = m.x;
        mag[2 * h + 1] = m.y;
        ang[2 * h] = a.x;
        ang[2 * h + 1] = a.y;
    }
}

// Gradient magnitude and angle at image row yy, columns x .. x+3, from a shared plane of pitch P
// (ctr points at (yy, x); the column left of x and right of x + 3 and the rows above and below are
// held): dx = right - left, dy = above - below, both zero on the image border as in the reference.
// One border test per group of four columns; the per-column test only where the group touches it.
template <int P>
__device__ __forceinline__ void grad4(const float* ctr, int yy, int x, int R, int C, float (&mg)[4], float (&an)[4]) {
    const float4 cc = *reinterpret_cast<const float4*>(ctr);
    const float4 up = *reinterpret_cast<const float4*>(ctr - P);
    const float4 dn = *reinterpret_cast<const float4*>(ctr + P);
    const float lf = ctr[-1], rt = ctr[4];
    float dx[4] = {__fsub_rn(cc.y, lf), __fsub_rn(cc.z, cc.x), __fsub_rn(cc.w, cc.y), __fsub_rn(rt, cc.z)};
    float dy[4] = {__fsub_rn(up.x, dn.x), __fsub_rn(up.y, dn.y), __fsub_rn(up.z, dn.z), __fsub_rn(up.w, dn.w)};
    if (!(yy > 0 && yy < R - 1 && x > 0 && x + 4 < C)) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (!(yy > 0 && yy < R - 1 && x + k > 0 && x + k < C - 1)) dx[k] = dy[k] = 0.f;
    }
    fast_grad4(dx, dy, mg, an);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}


// bounded waits on a shared-memory mbarrier (TMA completion)
constexpr long long TILE_TIMEOUT = 2000000000ll;   // cycles (about a second) for one TMA copy

__device__ __forceinline__ uint32_t s_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool s_mbar_test(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(s_addr(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits (bounded) for one row block; every thread waits, then the CTA agrees on the outcome.
__device__ __forceinline__ bool s_mbar_wait(uint64_t* b, uint32_t parity) {
    bool ok = s_mbar_test(b, parity);
    if (!ok) {
        const long long t0 = clock64();
        while (!(ok = s_mbar_test(b, parity)) && clock64() - t0 < TILE_TIMEOUT) {
        }
    }
    return ok;
}

// ------------------------------------------------------------------------------------------------
// Per-layer tiled kernels (float32 path), 128 x 32 outputs per CTA:
//   k_layer<I, RAD(I), false>  L_I of one octave from L_{I-1}: the same pair blurs and gradient as
//                              the layer groups (bit-identical results), DoG, gradient of L_{I-1},
//                              L_{I-1}[::2, ::2]
//   k_layer<0, 5, true>        the octave-0 base: the 2x bilinear upsample of the uint8 image
//                              (the reference's float32 rounding, gsift.py:90-102) computed while the
//                              tile loads, from per-row / per-column source tables, blurred with tap
//                              set 0
// The input tile (16 columns and r rows of reflect-101 halo) arrives by 16-byte cp.async, the
// vertical pass keeps an 8-row sliding window of column pairs in registers, the horizontal pass
// reads the row-pair interleaved vertical outputs. No ring buffers: 3-4 CTAs per SM.
constexpr int LX = 128, LNT = 256;   // tile width, threads; the tile height LY is a template parameter
constexpr int LIN_C = LX + 32;   // input tile columns (16 of halo on each side)
constexpr int LIN_W = LX + 40;   // input tile pitch (floats): rows 2 apart differ by 64 bytes mod 128
constexpr int LT2_W = LX + 34;   // row-pair tile pitch (float2): 16 bytes past a multiple of 128, so
                                 // row pairs p and p + 1 start in opposite 16-byte bank groups

struct LayerArgs {
    const float* src;   // L_{I-1}, R x C
    const uint8_t* img; // base: uint8 image ih x iw, row pitch img_stride
    const ImageSlot* slot;   // base: the image's address is read here (null: img)
    int img_stride, ih, iw;
    int R, C, P;        // octave rows, columns, row pitch of every plane
    float* dst;         // L_I or null
    float* dog;         // L_I - L_{I-1}
    float2* grad;       // gradient (magnitude, angle) of L_{I-1} or null
    float* down;        // L_{I-1}[::2, ::2] or null
    int down_pitch;
    int* err;           // set to 1 when the tile's TMA copy does not complete in time
};

// shared memory: the input tile (LIN_W floats per row), the row-pair tile, the TMA mbarrier
template <int r, int LY>
constexpr int layer_bar_off() {
    return (LY + 2 * r) * LIN_W * 4 + (LY / 2) * LT2_W * 8;
}
template <int r, int LY>
constexpr int layer_smem() {
    return layer_bar_off<r, LY>() + 16;
}

// The input tile (rows y0 - r .., columns x0 - 16 .., reflect-101 outside the plane) by
// per-thread cp.async (the caller commits and waits)
template <int r, int LY>
__device__ __forceinline__ void layer_load_cp(const LayerArgs& a, float* __restrict__ s_in, int x0, int y0) {
    constexpr int IH = LY + 2 * r;
    const int tid = threadIdx.x;
    if (x0 >= 16 && x0 + LX + 16 <= a.C) {
        // eight lanes per row (the mirrored row address once per row), five 16-byte copies a lane
        static_assert(LIN_C / 4 == 40, "five copies of eight lanes per row");
        for (int row = tid >> 3; row < IH; row += LNT / 8) {
            const float* g = a.src + (size_t)mir(y0 - r + row, a.R) * a.P + (x0 - 16);
            float* d = s_in + row * LIN_W;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int q = 4 * ((tid & 7) + 8 * k);
                cp_async16(d + q, g + q);
            }
        }
    } else {
        for (int i = tid; i < IH * LIN_C; i += LNT) {
            const int row = i / LIN_C, col = i - row * LIN_C;
            const float* g = a.src + (size_t)mir(y0 - r + row, a.R) * a.P + mir(x0 - 16 + col, a.C);
            cp_async4(s_in + row * LIN_W + col, g);
        }
    }
}

// Whether a tile's input lies inside the plane (no reflected row or column): such tiles arrive by
// one 2-D tensor copy of LIN_W x (LY + 2r) floats (the copy's last 8 columns are not read and may
// lie outside the plane, where the copy fills zeros)
template <int r, int LY>
__device__ __forceinline__ bool layer_tile_inside(const LayerArgs& a, int x0, int y0) {
    return y0 >= r && y0 + LY + r <= a.R && x0 >= 16 && x0 + LX + 16 <= a.C;
}
// thread 0: the tile's tensor copy into s_in, completion (bytes) on bar
template <int r, int LY>
__device__ __forceinline__ void layer_tma_issue(const CUtensorMap* tm, float* s_in, uint64_t* bar, int x0, int y0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s_addr(bar)),
                 "r"((LY + 2 * r) * LIN_W * 4)
                 : "memory");
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(s_addr(s_in)),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(x0 - 16), "r"(y0 - r), "r"(s_addr(bar))
        : "memory");
}

// The passes of one tile once its input (s_in) is in shared memory: vertical pass into the
// row-pair tile t2, then the horizontal pass and the epilogue (L_I, DoG, gradient, downsample).
template <int TS, int r, bool BASE, int LY>
__device__ __forceinline__ void layer_compute(const LayerArgs& a, const float* __restrict__ s_in,
                                              float2* __restrict__ t2, int x0, int y0) {
    constexpr int d = r & 1;
    constexpr int NPAIR = (LX + 2 * r + 2 * d) / 2;
    const int tid = threadIdx.x;
    // vertical pass: column pair cp (V columns 2cp, 2cp+1 = image columns x0 - r - d + 2cp ..),
    // output rows 8g .. 8g + 7; stored row-pair interleaved at t2 index (V column + d)
    float2 w[r + 1];
    load_taps<TS, r>(w);
    for (int it = tid; it < NPAIR * (LY / 8); it += LNT) {
        const int cp = it % NPAIR, g = it / NPAIR;
        const float* base = s_in + (8 * g) * LIN_W + (16 - r - d + 2 * cp);
        float2 x[8 + 2 * r];
#pragma unroll
        for (int k = 0; k < 8 + 2 * r; ++k) x[k] = *reinterpret_cast<const float2*>(base + k * LIN_W);
#pragma unroll
        for (int sp = 0; sp < 4; ++sp) {
            const float2 o0 = blur_pairs_w<r>(x + 2 * sp, w), o1 = blur_pairs_w<r>(x + 2 * sp + 1, w);
            float2* dst = t2 + (4 * g + sp) * LT2_W + 2 * cp + d;
            dst[0] = make_float2(o0.x, o1.x);
            dst[1] = make_float2(o0.y, o1.y);
        }
    }
    __syncthreads();
    // horizontal pass: row pair p, output columns c .. c+3 (t2 indices c + 2d .. c + 2d + 3 + 2r).
    // A warp covers row pairs p, p + 1 x 64 columns. 16-byte loads are served 8 lanes at a time:
    // in each group of 8 lanes, four read row pair p and four row pair p + 1 (columns 4 apart, a
    // 32-byte stride: one bank parity per row pair, opposite parities by the pitch), so the 8
    // lanes cover all 32 banks once
    static_assert(LX == 128 && (LY / 2) % 2 == 0 && LNT % 32 == 0, "horizontal pass mapping");
    // Fast path for tiles whose outputs and gradient neighbourhoods lie inside the plane (uniform per
    // CTA): no per-row bounds or border tests and 32-bit offsets. Same arithmetic as the general path
    // below, so the same bits.
    bool fast = (long long)a.R * a.P < (1ll << 31) && x0 + LX <= a.P && y0 + LY <= a.R;
    if (!BASE) fast = fast && (!a.grad || (y0 >= 1 && y0 + LY <= a.R - 1 && x0 >= 1 && x0 + LX < a.C));
    if (fast) {
        for (int it = tid; it < (LY / 2) * (LX / 4); it += LNT) {
            const int wi = it >> 5, l = it & 31;
            const int p = 2 * (wi >> 1) + ((l >> 2) & 1), c = 64 * (wi & 1) + 4 * ((l & 3) + 4 * (l >> 3));
            const int y = y0 + 2 * p, x = x0 + c;
            const float4* src = reinterpret_cast<const float4*>(t2 + p * LT2_W + c + 2 * d);
            float2 yv[4 + 2 * r];
#pragma unroll
            for (int k = 0; k < 2 + r; ++k) {
                const float4 v = src[k];
                yv[2 * k] = make_float2(v.x, v.y);
                yv[2 * k + 1] = make_float2(v.z, v.w);
            }
            float2 o[4];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) o[cc] = blur_pairs_w<r>(yv + cc, w);
            const int at0 = y * a.P + x;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int at = at0 + h * a.P;
                const float4 lv = h ? make_float4(o[0].y, o[1].y, o[2].y, o[3].y)
                                    : make_float4(o[0].x, o[1].x, o[2].x, o[3].x);
                if (BASE) {
                    *reinterpret_cast<float4*>(a.dst + at) = lv;
                    continue;
                }
                const float* ctr = s_in + (2 * p + h + r) * LIN_W + 16 + c;   // L_{I-1} at (y + h, x)
                const float4 pv = *reinterpret_cast<const float4*>(ctr);
                *reinterpret_cast<float4*>(a.dog + at) = make_float4(lv.x - pv.x, lv.y - pv.y, lv.z - pv.z, lv.w - pv.w);
                if (a.dst) *reinterpret_cast<float4*>(a.dst + at) = lv;
                if (a.grad) {
                    const float4 up = *reinterpret_cast<const float4*>(ctr - LIN_W);
                    const float4 dn = *reinterpret_cast<const float4*>(ctr + LIN_W);
                    const float lf = ctr[-1], rt = ctr[4];
                    const float dx[4] = {__fsub_rn(pv.y, lf), __fsub_rn(pv.z, pv.x), __fsub_rn(pv.w, pv.y),
                                         __fsub_rn(rt, pv.z)};
                    const float dy[4] = {__fsub_rn(up.x, dn.x), __fsub_rn(up.y, dn.y), __fsub_rn(up.z, dn.z),
                                         __fsub_rn(up.w, dn.w)};
                    float mg[4], an[4];
                    fast_grad4(dx, dy, mg, an);
                    st_grad4(a.grad + at, mg, an);
                }
                if (a.down && h == 0) {   // y is even: y0 and 2p are
                    float* o2 = a.down + (y >> 1) * a.down_pitch + (x >> 1);
                    o2[0] = pv.x;
                    o2[1] = pv.z;
                }
            }
        }
        return;
    }
    for (int it = tid; it < (LY / 2) * (LX / 4); it += LNT) {
        const int wi = it >> 5, l = it & 31;
        const int p = 2 * (wi >> 1) + ((l >> 2) & 1), c = 64 * (wi & 1) + 4 * ((l & 3) + 4 * (l >> 3));
        const int y = y0 + 2 * p, x = x0 + c;
        if (y >= a.R || x >= a.C) continue;
        const float4* src = reinterpret_cast<const float4*>(t2 + p * LT2_W + c + 2 * d);
        float2 yv[4 + 2 * r];
#pragma unroll
        for (int k = 0; k < 2 + r; ++k) {
            const float4 v = src[k];
            yv[2 * k] = make_float2(v.x, v.y);
            yv[2 * k + 1] = make_float2(v.z, v.w);
        }
        float2 o[4];
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) o[cc] = blur_pairs_w<r>(yv + cc, w);   // (row y, row y+1) at column x+cc
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int yy = y + h;
            if (yy >= a.R) break;
            // x < C and x % 4 = 0: the four columns lie inside the pitch
            const float4 lv = h ? make_float4(o[0].y, o[1].y, o[2].y, o[3].y)
                                : make_float4(o[0].x, o[1].x, o[2].x, o[3].x);
            const size_t at = (size_t)yy * a.P + x;
            if (BASE) {
                *reinterpret_cast<float4*>(a.dst + at) = lv;
                continue;
            }
            const float* ctr = s_in + (2 * p + h + r) * LIN_W + 16 + c;   // L_{I-1} at (yy, x)
            const float4 pv = *reinterpret_cast<const float4*>(ctr);
            *reinterpret_cast<float4*>(a.dog + at) = make_float4(lv.x - pv.x, lv.y - pv.y, lv.z - pv.z, lv.w - pv.w);
            if (a.dst) *reinterpret_cast<float4*>(a.dst + at) = lv;
            if (a.grad) {
                float mg[4], an[4];
                grad4<LIN_W>(ctr, yy, x, a.R, a.C, mg, an);
                st_grad4(a.grad + at, mg, an);
            }
            if (a.down && !(yy & 1)) {
                float* o2 = a.down + (size_t)(yy >> 1) * a.down_pitch + (x >> 1);
                o2[0] = pv.x;
                if (x + 2 < a.C) o2[1] = pv.z;
            }
        }
    }
}


template <int TS, int r, bool BASE, int LY>
__global__ void __launch_bounds__(LNT, r <= 10 ? 4 : 3) k_layer(const __grid_constant__ CUtensorMap tm, LayerArgs a,
                                                                int use_tma) {
    constexpr int d = r & 1;
    constexpr int IH = LY + 2 * r;
    constexpr int NPAIR = (LX + 2 * r + 2 * d) / 2;
    static_assert(layer_bar_off<r, LY>() % 16 == 0, "mbarrier alignment");
    extern __shared__ __align__(128) float sm[];
    float* s_in = sm;
    float2* t2 = reinterpret_cast<float2*>(sm + IH * LIN_W);
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * LX, y0 = blockIdx.y * LY;
    // input rows y0 - r .. y0 + LY + r - 1, columns x0 - 16 .. x0 + LX + 15 (reflect-101 outside)
    if (BASE) {
        // Source row / column pairs (iy, ny), (ix, nx) of every tile row / column (reflect-101 on
        // the upsampled grid). The source block they reach is staged once as scaled floats p, the
        // row-interpolated values vc = 0.75 p[iy] + 0.25 p[ny] are formed for every tile row over the
        // block's columns, and each upsampled sample is 0.75 vc[ix] + 0.25 vc[nx], four columns per
        // thread (gsift.py:90-102 rounding). Tables and vc live in the row-pair area and p in the
        // input tile until the vertical pass needs them. A block larger than the staging window
        // (mirror images of a tiny image) takes the per-sample global path.
        constexpr int VCW = 96, SRW = IH / 2 + 4;
        static_assert(!BASE || (2 * IH + 2 * LIN_C) * 4 + IH * VCW * 4 + 16 <= (LY / 2) * LT2_W * 8,
                      "base tables must fit the row-pair area");
        static_assert(!BASE || (SRW * VCW <= IH * LIN_W && IH % 2 == 0), "staged source block");
        int* ry = reinterpret_cast<int*>(t2);   // iy of tile row i, then ny
        int* rn = ry + IH;
        int* cxs = rn + IH;                      // ix of tile column c, then nx (16-byte aligned)
        int* cns = cxs + LIN_C;
        float* vcs = reinterpret_cast<float*>(cns + LIN_C);
        int* box = reinterpret_cast<int*>(vcs + IH * VCW);   // source row min / max, column min / max
        float* ps = s_in;
        const uint8_t* const img = a.slot ? a.slot->img : a.img;
        if (tid < 4) box[tid] = (tid & 1) ? -1 : 0x7fffffff;
        __syncthreads();
        for (int i0 = 0; i0 < IH + LIN_C; i0 += LNT) {
            const int i = i0 + tid;
            int lo = 0x7fffffff, hi = -1, clo = 0x7fffffff, chi = -1;
            if (i < IH) {
                const int Y = mir(y0 - r + i, a.R), iy = Y >> 1;
                const int ny = (Y & 1) ? min(iy + 1, a.ih - 1) : max(iy - 1, 0);
                ry[i] = iy;
                rn[i] = ny;
                lo = min(iy, ny);
                hi = max(iy, ny);
            } else if (i < IH + LIN_C) {
                const int c = i - IH, X = mir(x0 - 16 + c, a.C), ix = X >> 1;
                const int nx = (X & 1) ? min(ix + 1, a.iw - 1) : max(ix - 1, 0);
                cxs[c] = ix;
                cns[c] = nx;
                clo = min(ix, nx);
                chi = max(ix, nx);
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            clo = __reduce_min_sync(0xffffffffu, clo);
            chi = __reduce_max_sync(0xffffffffu, chi);
            if ((tid & 31) == 0) {
                if (hi >= 0) {
                    atomicMin(&box[0], lo);
                    atomicMax(&box[1], hi);
                }
                if (chi >= 0) {
                    atomicMin(&box[2], clo);
                    atomicMax(&box[3], chi);
                }
            }
        }
        __syncthreads();
        const int sy0 = box[0], nsr = box[1] - box[0] + 1, sx0 = box[2], nsx = box[3] - box[2] + 1;
        const float sc = (float)(1.0 / 255.0);
        if (nsr <= SRW && nsx <= VCW) {
            for (int row = tid >> 5; row < nsr; row += LNT / 32) {
                const uint8_t* src = img + (size_t)(sy0 + row) * a.img_stride + sx0;
                for (int k = tid & 31; k < nsx; k += 32) ps[row * VCW + k] = __fmul_rn((float)__ldg(src + k), sc);
            }
            __syncthreads();
            for (int i = tid; i < IH * (VCW / 4); i += LNT) {
                const int row = i / (VCW / 4), q = 4 * (i - row * (VCW / 4));
                if (q >= nsx) continue;
                const float4 p0 = *reinterpret_cast<const float4*>(ps + (ry[row] - sy0) * VCW + q);
                const float4 p1 = *reinterpret_cast<const float4*>(ps + (rn[row] - sy0) * VCW + q);
                float4 v;
                v.x = __fadd_rn(__fmul_rn(0.75f, p0.x), __fmul_rn(0.25f, p1.x));
                v.y = __fadd_rn(__fmul_rn(0.75f, p0.y), __fmul_rn(0.25f, p1.y));
                v.z = __fadd_rn(__fmul_rn(0.75f, p0.z), __fmul_rn(0.25f, p1.z));
                v.w = __fadd_rn(__fmul_rn(0.75f, p0.w), __fmul_rn(0.25f, p1.w));
                *reinterpret_cast<float4*>(vcs + row * VCW + q) = v;
            }
            __syncthreads();
            // Tiles whose columns reflect at no image or source edge: column X = x0 - 16 + q + k
            // samples source columns X / 2 and X / 2 -+ 1 in a fixed pattern, so four outputs take
            // four consecutive row-interpolated values (the same products and sums as the tables)
            if (x0 >= 18 && x0 + LX + 15 <= a.C - 3 && sx0 == (x0 - 16) / 2 - 1) {
                for (int i = tid; i < IH * (LIN_C / 4); i += LNT) {
                    const int row = i / (LIN_C / 4), m = i - row * (LIN_C / 4);
                    const float* vr = vcs + row * VCW + 2 * m;   // source columns X / 2 - 1 .. + 2
                    const float2 lo = *reinterpret_cast<const float2*>(vr);
                    const float2 hi = *reinterpret_cast<const float2*>(vr + 2);
                    const float a1 = __fmul_rn(0.75f, lo.y), a2 = __fmul_rn(0.75f, hi.x);
                    float4 u;
                    u.x = __fadd_rn(a1, __fmul_rn(0.25f, lo.x));
                    u.y = __fadd_rn(a1, __fmul_rn(0.25f, hi.x));
                    u.z = __fadd_rn(a2, __fmul_rn(0.25f, lo.y));
                    u.w = __fadd_rn(a2, __fmul_rn(0.25f, hi.y));
                    *reinterpret_cast<float4*>(s_in + row * LIN_W + 4 * m) = u;
                }
            } else {
            for (int i = tid; i < IH * (LIN_C / 4); i += LNT) {
                const int row = i / (LIN_C / 4), q = 4 * (i - row * (LIN_C / 4));
                const int4 ix = *reinterpret_cast<const int4*>(cxs + q);
                const int4 nx = *reinterpret_cast<const int4*>(cns + q);
                const float* v = vcs + row * VCW - sx0;
                float4 u;
                u.x = __fadd_rn(__fmul_rn(0.75f, v[ix.x]), __fmul_rn(0.25f, v[nx.x]));
                u.y = __fadd_rn(__fmul_rn(0.75f, v[ix.y]), __fmul_rn(0.25f, v[nx.y]));
                u.z = __fadd_rn(__fmul_rn(0.75f, v[ix.z]), __fmul_rn(0.25f, v[nx.z]));
                u.w = __fadd_rn(__fmul_rn(0.75f, v[ix.w]), __fmul_rn(0.25f, v[nx.w]));
                *reinterpret_cast<float4*>(s_in + row * LIN_W + q) = u;
            }
            }
        } else {
            for (int i = tid; i < IH * LIN_C; i += LNT) {
                const int row = i / LIN_C, col = i - row * LIN_C;
                const uint8_t* r0 = img + (size_t)ry[row] * a.img_stride;
                const uint8_t* r1 = img + (size_t)rn[row] * a.img_stride;
                const int ix = cxs[col], nx = cns[col];
                const float vc = __fadd_rn(__fmul_rn(0.75f, __fmul_rn((float)__ldg(r0 + ix), sc)),
                                           __fmul_rn(0.25f, __fmul_rn((float)__ldg(r1 + ix), sc)));
                const float vn = __fadd_rn(__fmul_rn(0.75f, __fmul_rn((float)__ldg(r0 + nx), sc)),
                                           __fmul_rn(0.25f, __fmul_rn((float)__ldg(r1 + nx), sc)));
                s_in[row * LIN_W + col] = __fadd_rn(__fmul_rn(0.75f, vc), __fmul_rn(0.25f, vn));
            }
        }
    } else if (use_tma && (s_addr(s_in) & 127) == 0 && layer_tile_inside<r, LY>(a, x0, y0)) {
        // an interior tile: one tensor copy, completion on an mbarrier
        uint64_t* bar = reinterpret_cast<uint64_t*>(reinterpret_cast<char*>(sm) + layer_bar_off<r, LY>());
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s_addr(bar)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (tid == 0) layer_tma_issue<r, LY>(&tm, s_in, bar, x0, y0);
        if (__syncthreads_or(!s_mbar_wait(bar, 0))) {
            // the copy did not land in time: flag it, give it one more bounded wait (so that no copy
            // into this CTA's shared memory is left in flight when possible) and leave the tile
            if (tid == 0) atomicExch(a.err, 1);
            s_mbar_wait(bar, 0);
            return;
        }
    } else {
        layer_load_cp<r, LY>(a, s_in, x0, y0);
    }
    cp_commit();
    cp_wait_all();
    __syncthreads();
    layer_compute<TS, r, BASE, LY>(a, s_in, t2, x0, y0);
}

// Tensor map of a layer's source plane (C columns of pitch P) for the tile copies (box LIN_W x
// rows): needs the box inside the plane's extent; 0 when not possible (the tiles then load by
// cp.async)
int layer_tensor_map(CUtensorMap* tm, const float* src, int R, int C, int P, int rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc || (P & 3) != 0 || C < LIN_W || R < rows || (reinterpret_cast<uintptr_t>(src) & 15) != 0) return 0;
    const cuuint64_t dims[2] = {(cuuint64_t)C, (cuuint64_t)R};
    const cuuint64_t strides[1] = {(cuuint64_t)P * 4};
    const cuuint32_t box[2] = {(cuuint32_t)LIN_W, (cuuint32_t)rows};
    const cuuint32_t es[2] = {1, 1};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(src), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int TS, int r, bool BASE, int LY>
int32_t launch_layer_ly(const LayerArgs& a, cudaStream_t s) {
    static std::atomic<int> attr[64];
    FSB_TRY(smem_attr((const void*)k_layer<TS, r, BASE, LY>, layer_smem<r, LY>(), attr));
    static_assert(LY + 2 * r <= 256, "tensor copy box height");
    CUtensorMap tm;
    std::memset(&tm, 0, sizeof(tm));
    const int use_tma = !BASE && a.err ? layer_tensor_map(&tm, a.src, a.R, a.C, a.P, LY + 2 * r) : 0;
    dim3 grid((a.C + LX - 1) / LX, (a.R + LY - 1) / LY);
    k_layer<TS, r, BASE, LY><<<grid, LNT, layer_smem<r, LY>(), s>>>(tm, a, use_tma);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

// tile heights the autotuner chooses from (index 0 is the default)
constexpr int kTileHeights[3] = {32, 16, 64};

template <int TS, int r, bool BASE>
int32_t launch_layer_t(const LayerArgs& a, int variant, cudaStream_t s) {
    if constexpr (BASE) {   // the base tile's source tables need a tile height of at least 32
        return variant == 2 ? launch_layer_ly<TS, r, BASE, 64>(a, s) : launch_layer_ly<TS, r, BASE, 32>(a, s);
    } else {
        switch (variant) {
            case 1: return launch_layer_ly<TS, r, BASE, 16>(a, s);
            case 2: return launch_layer_ly<TS, r, BASE, 64>(a, s);
            default: return launch_layer_ly<TS, r, BASE, 32>(a, s);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Fused layer groups (float32 path): one persistent kernel computes consecutive layers of an
// octave for output tiles of 128 x 32 (or smaller ones for octaves that would leave SMs idle, see
// launch_group_small),
//   group 0: L1, L2, L3 from L0 -> DoG 0..2, gradients of L1..L3, L3 and L3[::2, ::2]
//   group 1: L4, L5 from L3     -> DoG 3, 4
// Every level is held in shared memory on the tile plus the halo the levels above it need (row
// halo GH, column halo GXH; recomputed per tile), so the intermediate layers never reach HBM:
// per octave pixel the two launches read L0 and L3 and write the five DoG planes, six gradient
// planes, L3 and the downsample (14.25 octave planes of traffic where five per-layer launches move
// 20.25). Halo values outside the image equal the reflect-101 mirror of the values inside: the
// blur of a mirror-symmetric signal is mirror-symmetric and the pair sums of blur_pairs_t commute,
// so each level reproduces the per-layer kernels' values bit for bit. The passes are the per-layer
// kernel's (8-row register window of column pairs; row-pair-interleaved horizontal pass), with
// the DoG / gradient epilogue of a level run by the horizontal pass of the level above it. One
// CTA per SM walks the tiles; the next tile's input arrives by cp.async while this one computes.
// tile and threads: the large tile has the least halo, the small ones the shortest chain of passes
template <int X, int Y, int T>
struct GTile {
    static constexpr int GX = X, GY = Y, GNT = T;
};
using GLarge = GTile<128, 32, 512>;
using GMid = GTile<64, 16, 384>;
using GSmall = GTile<32, 16, 256>;

__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }

// One level of a group: the output level (row halo Ho, column halo Xo) blurred with radius r from
// the level below (Hi, Xi). The vertical pass covers input columns VS .. VS + VW - 1 (VS even);
// column j of its output sits at float2 index j + E of a row pair, so the horizontal pass's
// 16-byte loads start on an even index.
template <class Tile, int Hi, int Xi, int Ho, int Xo, int r>
struct GLevel : Tile {
    using Tile::GX;
    using Tile::GY;
    static constexpr int HIN = Hi, XIN = Xi, HOUT = Ho, XOUT = Xo, RAD = r;
    static constexpr int NIN = GY + 2 * Hi, MIN = GX + 2 * Xi;     // input rows, columns (= pitch)
    static constexpr int NOUT = GY + 2 * Ho, MOUT = GX + 2 * Xo;   // output rows, columns (= pitch)
    static constexpr int ROFF = Hi - Ho - r;                       // input row of output row 0's first tap
    static constexpr int OFF = Xi - Xo - r;                        // input column of output column 0's first tap
    static constexpr int E = OFF & 1;
    static constexpr int VS = OFF - E;
    static constexpr int VW = (MOUT + 2 * r + E + 1) & ~1;
    static constexpr int VP = (VW + E + 1) & ~1;                   // float2 per row pair
    static constexpr int V_FLOATS = (NOUT / 2) * VP * 2;
    static constexpr int IN_FLOATS = NIN * MIN, OUT_FLOATS = NOUT * MOUT;
    static_assert(ROFF >= 0 && OFF >= 0 && Xi % 4 == 0 && Xo % 4 == 0, "level geometry");
    static_assert(VS + VW <= MIN, "vertical pass inside the input level");
};

template <int G, class Tile>
struct GSpec;
template <class Tile>
struct GSpec<0, Tile> {
    using A = GLevel<Tile, 20, 28, 15, 20, 5>;   // L0 -> L1
    using B = GLevel<Tile, 15, 20, 9, 12, 6>;    // L1 -> L2
    using C = GLevel<Tile, 9, 12, 1, 4, 8>;      // L2 -> L3 (halo 1: gradient of L3)
    static constexpr int BUF0 = (cmax(A::IN_FLOATS, cmax(B::V_FLOATS, C::V_FLOATS)) + 3) & ~3;   // L0 / V2 / V3
    static constexpr int BUF1 = (cmax(A::V_FLOATS, B::OUT_FLOATS) + 3) & ~3;                     // V1 / L2
    static constexpr int BUF2 = (cmax(A::OUT_FLOATS, C::OUT_FLOATS) + 3) & ~3;                   // L1 / L3
};
template <class Tile>
struct GSpec<1, Tile> {
    using A = GLevel<Tile, 23, 28, 13, 16, 10>;   // L3 -> L4
    using B = GLevel<Tile, 13, 16, 0, 0, 13>;     // L4 -> L5 (tile only)
    static constexpr int BUF0 = (cmax(A::IN_FLOATS, B::V_FLOATS) + 3) & ~3;   // L3 / V5
    static constexpr int BUF1 = (A::V_FLOATS + 3) & ~3;                       // V4
    static constexpr int BUF2 = (A::OUT_FLOATS + 3) & ~3;                     // L4
};
// two input buffers (this tile's, the next tile's) and the two others
template <int G, class Tile>
constexpr int group_smem() {
    return (2 * GSpec<G, Tile>::BUF0 + GSpec<G, Tile>::BUF1 + GSpec<G, Tile>::BUF2) * 4;
}
static_assert(group_smem<0, GLarge>() <= 227 * 1024 && group_smem<1, GLarge>() <= 227 * 1024, "group shared memory");
static_assert(group_smem<0, GMid>() <= 113 * 1024 && group_smem<0, GSmall>() <= 75 * 1024, "two and three per SM");

struct GroupArgs {
    const float* src;   // the group's input level, R x C
    int R, C, P;        // octave rows, columns, row pitch of every plane
    int tiles_x, n_tiles;
    float* dog[3];      // DoG planes of the group's layers
    float2* grad[3];    // group 0: gradients of L1, L2, L3
    float* dst;         // group 0: L3
    float* down;        // group 0: L3[::2, ::2] or null
    int down_pitch;
};

// input level of tile t (rows y0 - HIN .., columns x0 - XIN .., reflect-101 outside) by cp.async
template <class L>
__device__ __forceinline__ void g_load(const GroupArgs& a, int t, float* dst) {
    constexpr int GNT = L::GNT;
    const int y0 = (t / a.tiles_x) * L::GY, cx = (t % a.tiles_x) * L::GX - L::XIN;
    if (cx >= 0 && cx + L::MIN <= a.C) {
        // eight lanes per row (the mirrored row address once per row)
        for (int row = threadIdx.x >> 3; row < L::NIN; row += GNT / 8) {
            const float* g = a.src + (size_t)mir(y0 - L::HIN + row, a.R) * a.P + cx;
#pragma unroll
            for (int k = 0; k < (L::MIN / 4 + 7) / 8; ++k) {
                const int q = (threadIdx.x & 7) + 8 * k;
                if (q < L::MIN / 4) cp_async16(dst + row * L::MIN + 4 * q, g + 4 * q);
            }
        }
    } else {
        for (int i = threadIdx.x; i < L::NIN * L::MIN; i += GNT) {
            const int row = i / L::MIN, col = i - row * L::MIN;
            cp_async4(dst + row * L::MIN + col, a.src + (size_t)mir(y0 - L::HIN + row, a.R) * a.P + mir(cx + col, a.C));
        }
    }
}

// vertical pass of level L: thread item = (column pair, 8 output rows); the last group of a level
// whose height is not a multiple of 8 starts at row NOUT - 8 (rows it shares with the group before
// are written twice with the same values), so every load stays inside the input level. Only the
// level's rows below kmax and the columns its horizontal pass reads for output columns below jmax
// are computed (a tile that reaches past the image needs its level only to the halo beyond it).
template <int TS, class L>
__device__ __forceinline__ void g_vpass(const float* __restrict__ pin, float2* __restrict__ v, int kmax, int jmax) {
    constexpr int r = L::RAD, NQ = L::VW / 2, NG = (L::NOUT + 7) / 8, GNT = L::GNT;
    static_assert(L::NOUT >= 8 && L::NIN == L::NOUT + 2 * r + 2 * L::ROFF, "vertical pass rows");
    float2 w[r + 1];
    load_taps<TS, r>(w);
    const int qmax = jmax + 2 * r + L::E + 4;   // 2q below it: every column the needed items read
    for (int it = threadIdx.x; it < NQ * NG; it += GNT) {
        const int q = it % NQ, g = it / NQ;
        const int y8 = min(8 * g, L::NOUT - 8);
        if (y8 >= kmax || 2 * q >= qmax) continue;
        const float* base = pin + (y8 + L::ROFF) * L::MIN + L::VS + 2 * q;
        float2 x[8 + 2 * r];
#pragma unroll
        for (int k = 0; k < 8 + 2 * r; ++k) x[k] = *reinterpret_cast<const float2*>(base + k * L::MIN);
        float2* d = v + (y8 / 2) * L::VP + 2 * q + L::E;
#pragma unroll
        for (int sp = 0; sp < 4; ++sp) {
            const float2 o0 = blur_pairs_w<r>(x + 2 * sp, w), o1 = blur_pairs_w<r>(x + 2 * sp + 1, w);
            d[sp * L::VP] = make_float2(o0.x, o1.x);
            d[sp * L::VP + 1] = make_float2(o0.y, o1.y);
        }
    }
}

// horizontal pass of level L: thread item = (row pair, 4 columns); the level's rows go to `pout`
// (when not null) and epi(tile row of the upper row, tile column, upper row, lower row) runs for
// every item (it checks the tile bounds itself); items at rows from kmax or columns from jmax on
// are not needed and skipped
template <int TS, class L, class Epi>
__device__ __forceinline__ void g_hpass(const float2* __restrict__ v, float* __restrict__ pout, Epi epi, int kmax,
                                        int jmax) {
    constexpr int r = L::RAD, NC = L::MOUT / 4, NP = L::NOUT / 2, GNT = L::GNT;
    float2 w[r + 1];
    load_taps<TS, r>(w);
    for (int it = threadIdx.x; it < NP * NC; it += GNT) {
        const int p = it / NC, c = 4 * (it - p * NC);
        if (2 * p >= kmax || c >= jmax) continue;
        const float4* src = reinterpret_cast<const float4*>(v + p * L::VP + c + 2 * L::E);
        float2 yv[4 + 2 * r];
#pragma unroll
        for (int k = 0; k < 2 + r; ++k) {
            const float4 t = src[k];
            yv[2 * k] = make_float2(t.x, t.y);
            yv[2 * k + 1] = make_float2(t.z, t.w);
        }
        float2 o[4];
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) o[cc] = blur_pairs_w<r>(yv + cc, w);
        const float4 top = make_float4(o[0].x, o[1].x, o[2].x, o[3].x);
        const float4 bot = make_float4(o[0].y, o[1].y, o[2].y, o[3].y);
        if (pout) {
            *reinterpret_cast<float4*>(pout + (2 * p) * L::MOUT + c) = top;
            *reinterpret_cast<float4*>(pout + (2 * p + 1) * L::MOUT + c) = bot;
        }
        epi(2 * p - L::HOUT, c - L::XOUT, top, bot);
    }
}

// at image row yy, columns xx .. xx + 3: the DoG cur - prev and, with grad set, the gradient of
// prev (prev points at prev(yy, xx) in a shared level of pitch P; the same arithmetic as k_layer)
template <int P>
__device__ __forceinline__ void g_dog_grad(const GroupArgs& a, int yy, int xx, const float* prev, float4 cur,
                                           float* dog, float2* grad) {
    const float4 pv = *reinterpret_cast<const float4*>(prev);
    const size_t at = (size_t)yy * a.P + xx;   // xx is a multiple of 4 below C
    *reinterpret_cast<float4*>(dog + at) = make_float4(cur.x - pv.x, cur.y - pv.y, cur.z - pv.z, cur.w - pv.w);
    if (grad) {
        float mg[4], an[4];
        grad4<P>(prev, yy, xx, a.R, a.C, mg, an);
        st_grad4(grad + at, mg, an);
    }
}

// epilogue of a level: for the tile pixels of an item, DoG (this level - prev) and the gradient of
// prev, prev being the shared level (halo PH, PX, pitch P) below
template <class Tile, int PH, int PX, int P>
struct GEpi {
    const GroupArgs& a;
    int y0, x0;
    const float* prev;
    float* dog;
    float2* grad;
    __device__ __forceinline__ void operator()(int ty, int tx, float4 top, float4 bot) const {
        if (tx < 0 || tx >= Tile::GX || x0 + tx >= a.C) return;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = ty + h;
            if (t < 0 || t >= Tile::GY || y0 + t >= a.R) continue;
            g_dog_grad<P>(a, y0 + t, x0 + tx, prev + (PH + t) * P + PX + tx, h ? bot : top, dog, grad);
        }
    }
};

template <int G, class Tile>
__global__ void __launch_bounds__(Tile::GNT, Tile::GX == 128 ? 1 : Tile::GX == 64 ? 2 : 3) k_group(GroupArgs a) {
    constexpr int GX = Tile::GX, GY = Tile::GY, GNT = Tile::GNT;
    using Sp = GSpec<G, Tile>;
    using LA = typename Sp::A;
    extern __shared__ __align__(16) float sm[];
    float* b1 = sm + 2 * Sp::BUF0;
    float* b2 = b1 + Sp::BUF1;
    int t = blockIdx.x;
    if (t >= a.n_tiles) return;
    g_load<LA>(a, t, sm);
    cp_commit();
    for (int cur = 0; t < a.n_tiles; t += gridDim.x, cur ^= 1) {
        cp_wait_all();
        __syncthreads();   // this tile's input is in; every thread is done with the previous tile
        const int nt = t + gridDim.x;
        if (nt < a.n_tiles) g_load<LA>(a, nt, sm + (cur ^ 1) * Sp::BUF0);
        cp_commit();
        const int y0 = (t / a.tiles_x) * GY, x0 = (t % a.tiles_x) * GX;
        const int vy = min(GY, a.R - y0), vx = min(GX, a.C - x0);   // the tile's pixels inside the image
        float* b0 = sm + cur * Sp::BUF0;
        if constexpr (G == 0) {
            using LB = typename Sp::B;
            using LC = typename Sp::C;
            g_vpass<1, LA>(b0, reinterpret_cast<float2*>(b1), vy + 2 * LA::HOUT, vx + 2 * LA::XOUT);  // L0 -> V1
            __syncthreads();
            g_hpass<1, LA>(reinterpret_cast<const float2*>(b1), b2,                               // V1 -> L1
                           GEpi<Tile, LA::HIN, LA::XIN, LA::MIN>{a, y0, x0, b0, a.dog[0], nullptr},
                           vy + 2 * LA::HOUT, vx + 2 * LA::XOUT);
            __syncthreads();
            g_vpass<2, LB>(b2, reinterpret_cast<float2*>(b0), vy + 2 * LB::HOUT, vx + 2 * LB::XOUT);  // L1 -> V2
            __syncthreads();
            g_hpass<2, LB>(reinterpret_cast<const float2*>(b0), b1,                               // V2 -> L2
                           GEpi<Tile, LB::HIN, LB::XIN, LB::MIN>{a, y0, x0, b2, a.dog[1], a.grad[0]},
                           vy + 2 * LB::HOUT, vx + 2 * LB::XOUT);
            __syncthreads();
            g_vpass<3, LC>(b1, reinterpret_cast<float2*>(b0), vy + 2 * LC::HOUT, vx + 2 * LC::XOUT);  // L2 -> V3
            __syncthreads();
            g_hpass<3, LC>(reinterpret_cast<const float2*>(b0), b2,                               // V3 -> L3
                           GEpi<Tile, LC::HIN, LC::XIN, LC::MIN>{a, y0, x0, b1, a.dog[2], a.grad[1]},
                           vy + 2 * LC::HOUT, vx + 2 * LC::XOUT);
            __syncthreads();
            // gradient of L3, L3 and L3[::2, ::2] on the tile
            for (int it = threadIdx.x; it < GY * (GX / 4); it += GNT) {
                const int ty = it / (GX / 4), tx = 4 * (it - ty * (GX / 4));
                const int yy = y0 + ty, xx = x0 + tx;
                if (yy >= a.R || xx >= a.C) continue;
                const float* l3 = b2 + (LC::HOUT + ty) * LC::MOUT + LC::XOUT + tx;
                const float4 v = *reinterpret_cast<const float4*>(l3);
                float mg[4], an[4];
                grad4<LC::MOUT>(l3, yy, xx, a.R, a.C, mg, an);
                const size_t at = (size_t)yy * a.P + xx;
                st_grad4(a.grad[2] + at, mg, an);
                *reinterpret_cast<float4*>(a.dst + at) = v;
                if (a.down && !(yy & 1)) {
                    float* o2 = a.down + (size_t)(yy >> 1) * a.down_pitch + (xx >> 1);
                    o2[0] = v.x;
                    if (xx + 2 < a.C) o2[1] = v.z;
                }
            }
        } else {
            using LB = typename Sp::B;
            g_vpass<4, LA>(b0, reinterpret_cast<float2*>(b1), vy + 2 * LA::HOUT, vx + 2 * LA::XOUT);  // L3 -> V4
            __syncthreads();
            g_hpass<4, LA>(reinterpret_cast<const float2*>(b1), b2,                               // V4 -> L4
                           GEpi<Tile, LA::HIN, LA::XIN, LA::MIN>{a, y0, x0, b0, a.dog[0], nullptr},
                           vy + 2 * LA::HOUT, vx + 2 * LA::XOUT);
            __syncthreads();
            g_vpass<5, LB>(b2, reinterpret_cast<float2*>(b0), vy + 2 * LB::HOUT, vx + 2 * LB::XOUT);  // L4 -> V5
            __syncthreads();
            g_hpass<5, LB>(reinterpret_cast<const float2*>(b0), nullptr,                          // V5 -> L5
                           GEpi<Tile, LB::HIN, LB::XIN, LB::MIN>{a, y0, x0, b2, a.dog[1], nullptr},
                           vy + 2 * LB::HOUT, vx + 2 * LB::XOUT);
        }
    }
    cp_wait_all();
}

int sm_count() {
    static int n[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 148;
    if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n[dev] = 148;
    return n[dev];
}

template <int G, class Tile>
int32_t launch_group_t(GroupArgs a, cudaStream_t s) {
    static std::atomic<int> attr[64];
    FSB_TRY(smem_attr((const void*)k_group<G, Tile>, group_smem<G, Tile>(), attr));
    a.tiles_x = (a.C + Tile::GX - 1) / Tile::GX;
    a.n_tiles = a.tiles_x * ((a.R + Tile::GY - 1) / Tile::GY);
    const int resident = sm_count() * (Tile::GX == 128 ? 1 : Tile::GX == 64 ? 2 : 3);
    const int grid = a.n_tiles < resident ? a.n_tiles : resident;
    k_group<G, Tile><<<grid, Tile::GNT, group_smem<G, Tile>(), s>>>(a);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

// The group with tiles for small octaves: 32 x 16 while they all fit on the GPU at once, else 64 x 16. An
// octave of 240 x 320 is 24 tiles of 128 x 32 - 24 SMs, each six passes over 13 000 pixels of input,
// 17 us - or 150 tiles of 32 x 16 with 5 000 pixels each. 320 x 240: the groups 18.7 and 14.7 us a
// launch, now 10.9 and 9.6; the whole pyramid 147 -> 117 us.
template <int G>
int32_t launch_group_small(const GroupArgs& a, cudaStream_t s) {
    const long long small = (long long)((a.C + 31) / 32) * ((a.R + 15) / 16);
    return small <= 3ll * sm_count() ? launch_group_t<G, GSmall>(a, s) : launch_group_t<G, GMid>(a, s);
}

}  // namespace

int layer_tile_variants() { return 3; }
int layer_tile_height(int variant) { return kTileHeights[variant < 0 || variant > 2 ? 0 : variant]; }

// One layer of the float32 pyramid by the tiled per-layer kernel: L_layer from src (R x C, pitch P), tile
// height layer_tile_height(variant).
int32_t launch_layer_fast(int layer, const float* src, int R, int C, int P, float* dst, float* dog, float2* grad,
                          float* down, int down_pitch, int variant, int* err, cudaStream_t s) {
    LayerArgs a{};
    a.err = err;
    a.src = src;
    a.R = R;
    a.C = C;
    a.P = P;
    a.dst = dst;
    a.dog = dog;
    a.grad = grad;
    a.down = down;
    a.down_pitch = down_pitch;
    switch (layer) {
        case 1: return launch_layer_t<1, 5, false>(a, variant, s);
        case 2: return launch_layer_t<2, 6, false>(a, variant, s);
        case 3: return launch_layer_t<3, 8, false>(a, variant, s);
        case 4: return launch_layer_t<4, 10, false>(a, variant, s);
        case 5: return launch_layer_t<5, 13, false>(a, variant, s);
        default: set_error("layer %d out of range", layer); return FSB_ERR_ARG;
    }
}


// Layers 1..3 of a float32 octave by the fused group kernel: from L0 (src, R x C, pitch P), DoG planes
// 0..2 at dog, dog + RC, dog + 2RC, gradients of L1..L3 at grad (+ RC, + 2RC), L3 to l3 and
// L3[::2, ::2] to down (null: last octave). down must not alias src (other tiles still read it). small:
// the tiles for small octaves.
int32_t launch_group_lower(const float* src, int R, int C, int P, float* dog, float2* grad, float* l3, float* down,
                           int down_pitch, bool small, cudaStream_t s) {
    const long long RC = (long long)R * P;
    GroupArgs a{};
    a.src = src;
    a.R = R;
    a.C = C;
    a.P = P;
    for (int k = 0; k < 3; ++k) {
        a.dog[k] = dog + k * RC;
        a.grad[k] = grad + k * RC;
    }
    a.dst = l3;
    a.down = down;
    a.down_pitch = down_pitch;
    return small ? launch_group_small<0>(a, s) : launch_group_t<0, GLarge>(a, s);
}

// Layers 4, 5 of a float32 octave by the fused group kernel: from L3 (src), DoG planes 3, 4 at
// dog3, dog3 + RC.
int32_t launch_group_upper(const float* src, int R, int C, int P, float* dog3, bool small, cudaStream_t s) {
    GroupArgs a{};
    a.src = src;
    a.R = R;
    a.C = C;
    a.P = P;
    a.dog[0] = dog3;
    a.dog[1] = dog3 + (long long)R * P;
    return small ? launch_group_small<1>(a, s) : launch_group_t<1, GLarge>(a, s);
}

// The float32 octave-0 base: blur (tap set 0, radius 5) of the 2x upsampled uint8 image.
int32_t launch_base_fast(const uint8_t* img, const ImageSlot* slot, int stride, int ih, int iw, int P, float* dst,
                         int variant, cudaStream_t s) {
    LayerArgs a{};
    a.img = img;
    a.slot = slot;
    a.img_stride = stride;
    a.ih = ih;
    a.iw = iw;
    a.R = 2 * ih;
    a.C = 2 * iw;
    a.P = P;
    a.dst = dst;
    return launch_layer_t<0, 5, true>(a, variant, s);
}

}  // namespace fsb
