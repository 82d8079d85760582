// The descriptor's walk over the pixels of a rotated unit square (also compiled for the host, where it is
// compared with the squares' definition).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifndef FSB_HD
#ifdef __CUDACC__
#define FSB_HD __host__ __device__ __forceinline__
#else
#define FSB_HD inline
#endif
#endif

namespace fsb {

FSB_HD uint32_t sq_bits(float v) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(v);
#else
    uint32_t u;
    memcpy(&u, &v, 4);
    return u;
#endif
}

// The pixels of one unit square (R', C') of the rotated bin grid, row by row: pixel (i, j) of the
// keypoint's window lies in the square when 0 <= j sin + i cos + 1.5 - R' < 1 and
// 0 <= j cos - i sin + 1.5 - C' < 1. Each row's column interval is solved in closed form, widened by
// SQ_BIN in bin units and SQ_PX in pixels, which cover the rounding of both this solve and the
// sample's own bin position (a few 1e-6 bins, 1e-7 |j| pixels); the sample's own test decides, so a
// wider interval changes no result. One step per call and no loop inside, so that a warp's lanes,
// each in its own square, stay converged: a step that opens an empty row yields no pixel.
constexpr float SQ_BIN = 2e-5f, SQ_PX = 0.01f, SQ_AMIN = 1e-10f;
constexpr float SQ_M = 12582912.f;   // 1.5 * 2^23: adding it rounds to an integer, held in the low bits
struct SquareWalk {
    float kl0, kl1, kh0, ml0, ml1, mh0;   // interval ends k0 + k1 i (both ends share the slope)
    float i, i1, j, j1, jmin, jmax;       // j, j1 hold SQ_M + column
    uint64_t row;                         // address of pixel (i, 0) less 8 times the bits of SQ_M

    FSB_HD void init(float sn, float cs, float Rf, float Cf, float hw, int ilo, int ihi, int jlo,
                     int jhi, const void* ctr, int pitch, bool on) {
        // a slope below SQ_AMIN is a row condition: its interval is everything or empty either way
        const float a = copysignf(fmaxf(fabsf(sn), SQ_AMIN), sn), b = copysignf(fmaxf(fabsf(cs), SQ_AMIN), cs);
        const float ia = 1.f / a, ib = 1.f / b;
        const float r0 = 1.5f - Rf, c0 = 1.5f - Cf;
        const float lo = -SQ_BIN, hi = 1.f + SQ_BIN;
        // j in [(lo - r0 - i cos) / a, (hi - r0 - i cos) / a], ends swapped for a negative slope; the
        // first column is the end rounded up and the last one rounded down, as nearest of +- 0.5
        kl0 = ((a > 0.f ? lo : hi) - r0) * ia + (0.5f - SQ_PX);
        kh0 = ((a > 0.f ? hi : lo) - r0) * ia - (0.5f - SQ_PX);
        kl1 = -cs * ia;
        ml0 = ((b > 0.f ? lo : hi) - c0) * ib + (0.5f - SQ_PX);
        mh0 = ((b > 0.f ? hi : lo) - c0) * ib - (0.5f - SQ_PX);
        ml1 = sn * ib;
        // rows: i = hw^2 (r cos - c sin) at the square's corners
        float imin = 1e30f, imax = -1e30f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float iv = hw * hw * ((Rf + (float)(q >> 1) - 1.5f) * cs - (Cf + (float)(q & 1) - 1.5f) * sn);
            imin = fminf(imin, iv);
            imax = fmaxf(imax, iv);
        }
        const float sl = SQ_PX + 2.f * SQ_BIN * hw + 1e-6f * fmaxf(fabsf(imin), fabsf(imax));
        const int first = (int)ceilf(imin - sl), is = (ilo > first ? ilo : first) - 1;
        i = (float)is;
        i1 = on ? fminf((float)ihi, floorf(imax + sl)) : -1e30f;
        row = reinterpret_cast<uint64_t>(ctr) + 8ll * ((long long)is * pitch) - 8ull * sq_bits(SQ_M);
        jmin = (float)jlo;
        jmax = (float)jhi;
        j = SQ_M + 1.f;
        j1 = SQ_M;
    }
    // returns whether the walk stayed in its row
    FSB_HD bool step(int pitch) {
        j += 1.f;
        const bool stay = j <= j1;
        if (!stay) {
            i += 1.f;
            row += 8ll * pitch;
            j = fmaxf(fmaxf(fmaf(i, kl1, kl0), fmaf(i, ml1, ml0)), jmin) + SQ_M;
            j1 = fminf(fminf(fmaf(i, kl1, kh0), fmaf(i, ml1, mh0)), jmax) + SQ_M;
        }
        return stay;
    }
    FSB_HD bool alive() const { return i <= i1; }
    FSB_HD bool valid() const { return i <= i1 && j <= j1; }
    FSB_HD uint64_t pixel() const { return row + 8ull * sq_bits(j); }   // its address
};

}  // namespace fsb
