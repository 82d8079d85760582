"""The descriptor's pixel walk against the definition of its squares, on the host: for orientations along the
axes, the diagonals and next to them, windows cut by each border, centres outside the image and scales from a
fraction of a pixel to beyond the image, every pixel of the window that the sample's own test puts into a
square is walked by that square's lane exactly once and in row order, in the float32 and the float64 test.
(A walk may offer pixels of other squares; the sample's test drops them.)"""
import ctypes
import os
import subprocess

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fieldstitch_b200", "csrc")

HARNESS = r"""
#include <math.h>
#include <vector>
#include "square_walk.cuh"
using namespace fsb;
// 0, or 1 + the number of pixels missed, taken twice or out of order; out[0] pixels inside, out[1] offered
extern "C" long long walk(double px, double py, double scl, double ori, int rows, int cols, long long* out) {
    long long radl = llrint(3.0 * scl * 1.4142135623730951 * 5.0 * 0.5);
    const long long rmax = (long long)sqrt((double)rows * rows + (double)cols * cols);
    if (radl > rmax) radl = rmax;
    const int rad = (int)radl, pr = (int)rint(py), pc = (int)rint(px);
    const double hw = 3.0 * scl, t = ori * 0.017453292519943295, cos_d = cos(t) / hw, sin_d = sin(t) / hw;
    const float cs = (float)cos_d, sn = (float)sin_d;
    const int ilo = -rad > 1 - pr ? -rad : 1 - pr, ihi = rad < rows - 2 - pr ? rad : rows - 2 - pr;
    const int jlo = -rad > 1 - pc ? -rad : 1 - pc, jhi = rad < cols - 2 - pc ? rad : cols - 2 - pc;
    long long bad = 0;
    out[0] = out[1] = 0;
    const int nj = jhi - jlo + 1, ni = ihi - ilo + 1, pitch = (cols + 3) & ~3;
    std::vector<signed char> seen;
    for (int lane = 0; lane < 25; ++lane) {
        const int Rq = lane / 5 - 1, Cq = lane % 5 - 1;
        seen.assign(ni > 0 && nj > 0 ? (size_t)ni * nj : 0, 0);
        SquareWalk w;
        // an address of its own for each pixel: 8 bytes, the centre far above zero
        const uint64_t ctr = 1ull << 40;
        w.init(sn, cs, (float)Rq, (float)Cq, (float)hw, ilo, ihi, jlo, jhi, (const void*)ctr, pitch, true);
        int li = -1000000000, lj = 0;
        for (long long guard = 0; w.alive(); ++guard) {
            w.step(pitch);
            if (guard > 40000000) return -1;
            if (!w.valid()) continue;
            const int i = (int)w.i, j = (int)(w.j - SQ_M);
            if (i < ilo || i > ihi || j < jlo || j > jhi) { ++bad; continue; }          // would read outside
            if (w.pixel() != ctr + 8ll * ((long long)i * pitch + j)) ++bad;              // its address
            if (i < li || (i == li && j <= lj)) ++bad;                                   // row order
            li = i; lj = j;
            ++seen[(size_t)(i - ilo) * nj + (j - jlo)];
            ++out[1];
        }
        for (int i = ilo; i <= ihi; ++i)
            for (int j = jlo; j <= jhi; ++j) {
                const float fi = (float)i, fj = (float)j;
                const float rb = fj * sn + fi * cs + 1.5f, cb = fj * cs - fi * sn + 1.5f;
                const bool in_f = rb > -1.f && rb < 4.f && cb > -1.f && cb < 4.f && (int)floorf(rb) == Rq && (int)floorf(cb) == Cq;
                const double rd = ((double)j * sin_d + (double)i * cos_d + 2.0) - 0.5, cd = ((double)j * cos_d - (double)i * sin_d + 2.0) - 0.5;
                const bool in_d = rd > -1.0 && rd < 4.0 && cd > -1.0 && cd < 4.0 && (int)floor(rd) == Rq && (int)floor(cd) == Cq;
                const int n = seen[(size_t)(i - ilo) * nj + (j - jlo)];
                if ((in_f || in_d) && n != 1) ++bad;
                if (n > 1) ++bad;
                out[0] += in_f;
            }
    }
    return bad ? 1 + bad : 0;
}
"""


def test_every_pixel_of_a_square_once(tmp_path):
    src, so = tmp_path / "walk.cpp", tmp_path / "walk.so"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)],
                   check=True)
    f = ctypes.CDLL(str(so)).walk
    f.restype = ctypes.c_longlong
    f.argtypes = [ctypes.c_double] * 4 + [ctypes.c_int] * 2 + [ctypes.c_void_p]
    out = (ctypes.c_longlong * 2)()
    rng = np.random.default_rng(4)
    angles = [0.0, 90.0, 180.0, 270.0, 45.0, 135.0, 225.0, 315.0, 26.565051177077994, 1e-6, 359.999999, 89.9999, 90.0001, 0.01]
    rows, cols = 93, 121
    cases = [(x, y, s, a) for x in (0.0, 1.0, 60.5, cols - 2.0, cols - 1.0, -5.0, cols + 6.3) for y in (0.4, 46.0, rows - 1.5, rows + 3.0)
             for s in (0.05, 0.31, 1.0, 2.7) for a in angles]
    cases += [(x, y, s, a) for x in (3.0, 60.2) for y in (45.9,) for s in (6.0, 17.0, 1.0 / 3.0, 2.0 / 3.0) for a in angles]
    cases += [(rng.uniform(-8, cols + 8), rng.uniform(-8, rows + 8), float(np.exp(rng.uniform(np.log(0.05), np.log(5)))),
               rng.uniform(0, 360)) for _ in range(600)]
    inside = offered = 0
    for x, y, s, a in cases:
        ori = 360.0 - float(np.float32(a))
        if abs(ori - 360.0) < 1e-4:
            ori = 0.0
        bad = f(float(np.float32(x)), float(np.float32(y)), s, ori, rows, cols, out)
        assert bad == 0, (x, y, s, a, bad)
        inside += out[0]
        offered += out[1]
    assert inside > 300000 and offered < 1.1 * inside + 25 * len(cases)   # and few pixels are offered in vain
