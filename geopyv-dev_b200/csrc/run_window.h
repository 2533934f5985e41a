// run_window.h -- the run length of the run-layout solves and the planning of the
// coefficient windows they stage in shared memory (host and device; no CUDA
// header needed).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define GPV_HD __host__ __device__ __forceinline__
#else
#define GPV_HD inline
#endif

namespace gpv {
namespace {

constexpr int kRunK = 4;       // template pixels per run
constexpr int kRunMargin = 2;  // pixels a window reaches past the warped square

// Window row pitch in elements: a multiple of 4 (16-byte rows for cp.async)
// that is not a multiple of BANKS, the elements one row of shared-memory banks
// holds (32 floats, 16 doubles), so two bands' rows read by one warp start on
// different banks.  Lanes of a warp read consecutive columns of one row.
template <int BANKS>
GPV_HD int run_pitch(int ww) {
    const int p = (ww + 3) & ~3;
    return (p & (BANKS - 1)) ? p : p + 4;
}

// A window covering pixel indices [xlo, xhi] x [ylo, yhi] (clamped to the
// image) plus the taps and kRunMargin; false if it does not fit in cap
// elements (the margin is dropped when the window with it does not fit).  A
// warp that spans a large image plans more elements than an int holds.
template <int BANKS>
GPV_HD bool run_plan(int xlo, int xhi, int ylo, int yhi, int border, int cap, int &r0, int &c0, int &wh, int &ww, int &pitch) {
    for (int m = kRunMargin; m >= 0; m -= kRunMargin) {
        const int clo = xlo + border - 2 - m, chi = xhi + border + 3 + m;
        c0 = clo >= 0 ? (clo & ~3) : -(((-clo) + 3) & ~3);
        ww = ((chi + 1 - c0) + 3) & ~3;
        pitch = run_pitch<BANKS>(ww);
        r0 = ylo + border - 2 - m;
        wh = yhi + border + 3 + m + 1 - r0;
        if ((int64_t)pitch * wh <= cap) return true;
        if (m == 0) break;
    }
    return false;
}

}  // namespace
}  // namespace gpv
