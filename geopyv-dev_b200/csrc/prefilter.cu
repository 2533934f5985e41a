// prefilter.cu -- bi-quintic B-spline coefficients on the device.
//
// Reference: get_c (src/image.rs:252-327).  The reference replicate-pads the
// image by `border` (pad_replicate, :436-443), then for every row and then
// every column computes IFFT(FFT(line) / FFT(kernel)) with the zero-phase
// quintic kernel [11/20, 13/60, 1/120, 0, ..., 0, 1/120, 13/60]
// (build_kernel, :422-430), keeping the real part.
//
// That is a circular convolution with the periodised inverse filter
//     h_N[m] = (1/N) sum_j cos(2 pi j m / N) / K(2 pi j / N),
//     K(w)   = 11/20 + (13/30) cos w + (1/60) cos 2w,
// whose poles are z_i and 1/z_i with z_i + 1/z_i = w_i = -13 +- sqrt(105)
// (K = (w - w_1)(w - w_2) / 120 in w = z + 1/z), so by partial fractions
//     h[m] = A_1 z_1^|m| + A_2 z_2^|m|,  z_1 = -0.4306, z_2 = -0.0431,
// the sum of two decaying exponentials to either side: four first-order
// recursions (M. Unser, A. Aldroubi, M. Eden, "B-spline signal processing",
// IEEE Trans. Signal Process. 41, 1993, run them over whole lines; here they run
// over blocks with a lead-in).  A thread makes kQ outputs of one line: the
// recursions that come from the left start MT samples before them, those from
// the right MT samples after, so the taps dropped are those past |m| = MT of a
// direct filter: MT = 44 reproduces the FFT result to FP64 rounding (1e-14
// relative; see tests/test_prefilter_*), and an image whose coefficients are
// kept in FP32 only takes MT = 28 (dropped taps sum to 2.7e-10 of the largest
// input per pass, below FP32 rounding).  That is 14 FP64 multiply-adds per
// output and pass (MT = 28) against 57 of the direct filter this replaced,
// whose bound was the FP64 pipe (55 % of its peak); now the pixel loads' latency
// and the shared-memory reads bound it (FP64 pipe 17-25 %), so a warp has the
// loads of kAhead lines in flight and three blocks share an SM (80 registers).
// 4096^2 u16 207 -> 125 us, 2048^2 u8 63 -> 37, 911 x 1237 f64 with FP64
// coefficients 102 -> 28, 4096^2 f32 with FP64 coefficients 596 -> 276.  Groups of kQ outputs start at multiples of kQ
// of the padded line, so an output does not depend on how the rows are cut
// into launches and blocks.  Both passes run in one kernel (prefilter_fused):
// first along staged pixel rows, then down a ring of FP64 row-pass lines held in
// shared memory; the coefficients come out as FP32 (and optionally FP64),
// (h + 2b, w + 2b).  Images with a line shorter than 89 samples take every tap
// of the periodised filter, whose spectrum is evaluated in closed form once per
// line length N (the kernel's FFT in the reference), in two simple kernels
// through an FP64 row-pass buffer.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "internal.h"

namespace gpv {

namespace {
constexpr int kM = 44;             // lead-in of the recursions (FP64 coefficients)
constexpr int kM32 = 28;           // the same when the coefficients are kept in FP32 only
constexpr int kT = 2 * kM + 1;     // 89
constexpr int kGroups = 8;         // warps per block
constexpr int kQ = 16;             // outputs per thread

struct TapArg {
    double h[kT];  // h[k] multiplies x[j - mr + k]  (i.e. h_N[mr - k])
};

std::mutex g_taps_mu;
std::map<int64_t, Taps> g_taps;

// The two exponentials: poles z, weights A, and B = A z for the side that
// starts one sample off the centre.
struct Poles {
    double z1, z2, a1, a2, b1, b2;
    double t1;  // A_1 z_1^(kM32 + 1): what a tap past |m| = kM32 weighs
};

Poles poles() {
    const double w1 = -13.0 + std::sqrt(105.0), w2 = -13.0 - std::sqrt(105.0);
    Poles p;
    p.z1 = 2.0 / (w1 - std::sqrt(w1 * w1 - 4.0));
    p.z2 = 2.0 / (w2 - std::sqrt(w2 * w2 - 4.0));
    const double g = 120.0 / (w1 - w2);
    p.a1 = -g * p.z1 / (1.0 - p.z1 * p.z1);
    p.a2 = g * p.z2 / (1.0 - p.z2 * p.z2);
    p.b1 = p.a1 * p.z1;
    p.b2 = p.a2 * p.z2;
    p.t1 = p.a1 * std::pow(p.z1, kM32 + 1);
    return p;
}

// kQ outputs of a line from its 2 MT + kQ samples x(0 ..), output q at sample
// MT + q.  Both sides advance together (four independent chains); the fast
// pole needs W2 samples of lead-in only (0.0431^8 = 1.2e-11, ^13 = 1.8e-18).
// At MT = kM32 the slow pole's taps past |m| = MT, which the lead-in of the
// other outputs brings with it, are taken off again (the chain's state MT + 1
// samples back, times t1): every output is the filter of 2 MT + 1 taps, to FP64
// rounding, wherever it lies in its group.  A sample that is not finite stays in
// the chains to the group's end: false says that there is one, and the caller
// takes the group's outputs again tap by tap (tap_by_tap), so that it reaches
// |m| = MT and no farther.
template <int MT, class X>
__device__ __forceinline__ bool exponentials(X x, const Poles &c, double (&acc)[kQ]) {
    constexpr bool kCut = MT == kM32;
    constexpr int W2 = MT <= 28 ? 8 : 13;
    double p1 = 0.0, p2 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int q = 0; q < kQ; q++) acc[q] = 0.0;
#pragma unroll
    for (int k = 0; k < MT + kQ; k++) {
        {
            const double v = x(k);
            p1 = fma(c.z1, p1, v);
            if (k >= MT - W2) p2 = fma(c.z2, p2, v);
            if (kCut && k + 1 < kQ) acc[k + 1] = fma(-c.t1, p1, acc[k + 1]);
            const int q = k - MT;
            if (q >= 0) acc[q] = fma(c.a1, p1, fma(c.a2, p2, acc[q]));
        }
        const int sx = 2 * MT + kQ - 1 - k;
        if (sx > MT) {
            const double v = x(sx);
            s1 = fma(c.z1, s1, v);
            if (sx <= MT + kQ + W2) s2 = fma(c.z2, s2, v);
            if (kCut && sx > 2 * MT) acc[sx - 2 * MT - 1] = fma(-c.t1, s1, acc[sx - 2 * MT - 1]);
            const int q = sx - 1 - MT;
            if (q < kQ) acc[q] = fma(c.b1, s1, fma(c.b2, s2, acc[q]));
        }
    }
    return isfinite(p1) && isfinite(s1);
}

// One output tap by tap, x its sample.
template <int MT, class S>
__device__ __noinline__ double tap_by_tap(const S *x, int stride, double z1, double z2, double a1, double a2) {
    double acc = (a1 + a2) * (double)x[0];
#pragma unroll 1
    for (int m = 1; m <= MT; m++) {
        a1 *= z1;
        a2 *= z2;
        acc = fma(a1 + a2, (double)x[m * stride], fma(a1 + a2, (double)x[-m * stride], acc));
    }
    return acc;
}

// Both passes in one kernel.  A block owns a strip of kStrip padded columns
// [j0, j0 + kStrip) and a segment of output rows [i_beg, i_end).  It walks
// down the segment kStep rows at a time: the row pass of the next kStep
// padded rows (from pixel lines staged in shared memory) lands in a ring of
// FP64 lines that also holds the 2 MT lines before them, and the column pass
// of kStep outputs reads that ring.  The FP64 row-pass lines never leave the
// SM: DRAM sees the pixels (read once per strip; the halo columns of
// neighbouring strips come from L2) and the coefficients written.
//   row pass:    R[r] = the filter along X[r], X[r][jj] = px[r][clamp(jj mod cw - border, 0, w - 1)]
//   column pass: C[.][j] = the filter down R[clamp(i mod ch - border, 0, h - 1)][j]
constexpr int kStrip = 32;   // columns per block (one per lane in the column pass)
constexpr int kStep = 128;   // output rows per step (8 warps x kQ)
constexpr int kFusedThreads = kGroups * 32;
constexpr int kAhead = 4;    // pixel lines a warp has in flight while staging
static_assert(kStep == kGroups * kQ && kStrip == 2 * kQ, "one row-pass line per two threads, one output column per lane");

// Staged pixel line pitch (elements) for kPxW pixels: lanes of a warp read 32
// different lines at one column, so the pitch in 4-byte words is odd (an odd
// number of doubles for FP64 pixels).
template <typename P, int W>
__host__ __device__ constexpr int px_pitch() {
    return sizeof(P) == 8 ? (W | 1) : (((W * (int)sizeof(P) + 3) / 4) | 1) * 4 / (int)sizeof(P);
}

template <typename P, int MT>
struct Fused {
    static constexpr int kHalo = 2 * MT;
    static constexpr int kRing = kStep + kHalo;   // FP64 row-pass lines held
    static constexpr int kRingPitch = kStrip + 1;  // doubles
    static constexpr int kPxW = kStrip + kHalo;   // pixels per staged line
    static constexpr int kPxPitch = px_pitch<P, kPxW>();
    static constexpr size_t kRingBytes = sizeof(double) * kRing * kRingPitch;
    static constexpr size_t kSmem = kRingBytes + sizeof(P) * kStep * kPxPitch;
};

template <typename P, int MT>
__global__ void __launch_bounds__(kFusedThreads, 3) prefilter_fused(const P *__restrict__ px, int64_t h, int64_t w,
                                                                int64_t border, int64_t cw, int64_t ch, int64_t i_lo,
                                                                int64_t i_hi, int64_t seg, Poles poles,
                                                                float *__restrict__ c32, int64_t pitch32,
                                                                double *__restrict__ c64, int64_t pitch64) {
    using G = Fused<P, MT>;
    constexpr bool kAny = std::is_floating_point<P>::value;  // pixels may be NaN or infinite
    extern __shared__ double smem[];
    double *ring = smem;
    P *pxs = reinterpret_cast<P *>(reinterpret_cast<unsigned char *>(smem) + G::kRingBytes);
    const int64_t j0 = (int64_t)blockIdx.x * kStrip;
    const int64_t i_beg = i_lo + (int64_t)blockIdx.y * seg;  // a multiple of kQ, as i_lo and seg are
    const int64_t i_end = i_beg + seg < i_hi ? i_beg + seg : i_hi;
    if (i_beg >= i_end) return;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;

    // the strip's source columns, the same for every line: entry m of lane
    // l is staged column l + 32 m, its image column (-1 past the staged width)
    constexpr int kCols = (G::kPxW + 31) / 32;
    int csrc[kCols];
#pragma unroll
    for (int m = 0; m < kCols; m++) {
        const int sx = lane + 32 * m;
        int jj = (int)j0 - MT + sx;  // in [-MT, cw + kStrip + MT): one wrap at most (cw >= 2 MT + 1)
        jj = jj < 0 ? jj + (int)cw : (jj >= (int)cw ? jj - (int)cw : jj);
        const int c = jj - (int)border;
        csrc[m] = sx < G::kPxW ? (c < 0 ? 0 : (c > (int)w - 1 ? (int)w - 1 : c)) : -1;
    }
    // row pass of n padded rows (row0 + t) mod ch, t < n <= kStep, into ring
    // lines [dst, dst + n); the pixel lines are staged one per warp at a time
    auto produce = [&](int64_t row0, int n, int dst) {
        int base = (int)(row0 % ch);  // row0 >= -MT
        if (base < 0) base += (int)ch;
        // kAhead lines of a warp at a time, their loads together in flight
#pragma unroll 1
        for (int r0 = wid; r0 < n; r0 += kAhead * kGroups) {
            P v[kAhead][kCols];
#pragma unroll
            for (int a = 0; a < kAhead; a++) {
                const int rr = r0 + a * kGroups;
                int ii = base + min(rr, n - 1);
                while (ii >= (int)ch) ii -= (int)ch;
                const int r = min(max(ii - (int)border, 0), (int)h - 1);
                const P *src = px + (int64_t)r * w;
#pragma unroll
                for (int m = 0; m < kCols; m++)
                    if (csrc[m] >= 0) v[a][m] = src[csrc[m]];
            }
#pragma unroll
            for (int a = 0; a < kAhead; a++) {
                const int rr = r0 + a * kGroups;
                if (rr < n) {
                    P *d = pxs + rr * G::kPxPitch + lane;
#pragma unroll
                    for (int m = 0; m < kCols; m++)
                        if (csrc[m] >= 0) d[32 * m] = v[a][m];
                }
            }
        }
        __syncthreads();
        const int rr = (wid & 3) * 32 + lane, half = wid >> 2;
        if (rr < n) {
            const P *x = pxs + rr * G::kPxPitch + half * kQ;
            double acc[kQ];
            const bool fine = exponentials<MT>([&](int sx) { return (double)x[sx]; }, poles, acc);
            double *o = ring + (dst + rr) * G::kRingPitch + half * kQ;
#pragma unroll
            for (int q = 0; q < kQ; q++) o[q] = acc[q];
            if (kAny && !fine) {
#pragma unroll 1
                for (int q = 0; q < kQ; q++) o[q] = tap_by_tap<MT>(x + MT + q, 1, poles.z1, poles.z2, poles.a1, poles.a2);
            }
        }
        __syncthreads();
    };

    // the 2 MT lines before the first output
    produce(i_beg - MT, G::kHalo, 0);
    for (int64_t done = 0; done < i_end - i_beg; done += kStep) {
        const int n = (int)(i_end - i_beg - done < kStep ? i_end - i_beg - done : kStep);
        // whole groups of lines: the last group's recursions start past the segment's end
        produce(i_beg + MT + done, (n + kQ - 1) / kQ * kQ, G::kHalo);
        // column pass: lane = column, warp wid = outputs [wid kQ, wid kQ + kQ) of this step
        if (wid * kQ < n) {
            const double *x = ring + (wid * kQ) * G::kRingPitch + lane;
            double acc[kQ];
            const bool fine = exponentials<MT>([&](int sx) { return x[sx * G::kRingPitch]; }, poles, acc);
            const int64_t j = j0 + lane;
            if (j < cw) {
#pragma unroll
                for (int q = 0; q < kQ; q++) {
                    if (wid * kQ + q < n) {
                        const int64_t i = i_beg + done + wid * kQ + q;
                        c32[i * pitch32 + j] = (float)acc[q];
                        if (c64) c64[i * pitch64 + j] = acc[q];
                    }
                }
                if (kAny && !fine) {
#pragma unroll 1
                    for (int q = 0; q < kQ && wid * kQ + q < n; q++) {
                        const int64_t i = i_beg + done + wid * kQ + q;
                        const double v = tap_by_tap<MT>(x + (MT + q) * G::kRingPitch, G::kRingPitch, poles.z1, poles.z2, poles.a1, poles.a2);
                        c32[i * pitch32 + j] = (float)v;
                        if (c64) c64[i * pitch64 + j] = v;
                    }
                }
            }
        }
        if (n < kStep) break;  // the segment's last step
        __syncthreads();  // every column pass has read the ring
        // the last 2 MT lines become the first ones of the next step (n = kStep >= 2 MT: no overlap)
        for (int idx = tid; idx < G::kHalo * kStrip; idx += kFusedThreads) {
            const int rr = idx / kStrip, c = idx - rr * kStrip;
            ring[rr * G::kRingPitch + c] = ring[(kStep + rr) * G::kRingPitch + c];
        }
        __syncthreads();
    }
}

// Short lines (N < 89): every one of the N circulant taps, taps in global memory.
template <typename P>
__global__ void rowpass_small(const P *__restrict__ px, int64_t h, int64_t w, int64_t border, int64_t cw, int mr, int nt,
                              const double *__restrict__ taps, double *__restrict__ out) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= h * cw) return;
    const int64_t r = idx / cw, j = idx % cw;
    double acc = 0.0;
    for (int k = 0; k < nt; k++) {
        int64_t jj = (j - mr + k) % cw;
        if (jj < 0) jj += cw;
        int64_t c = jj - border;
        c = c < 0 ? 0 : (c > w - 1 ? w - 1 : c);
        acc = fma(taps[k], (double)px[r * w + c], acc);
    }
    out[idx] = acc;
}

__global__ void colpass_small(const double *__restrict__ rp, int64_t h, int64_t cw, int64_t ch, int64_t border, int mr,
                              int nt, const double *__restrict__ taps, float *__restrict__ c32, int64_t pitch32,
                              double *__restrict__ c64, int64_t pitch64) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ch * cw) return;
    const int64_t i = idx / cw, j = idx % cw;
    double acc = 0.0;
    for (int k = 0; k < nt; k++) {
        int64_t ii = (i - mr + k) % ch;
        if (ii < 0) ii += ch;
        int64_t r = ii - border;
        r = r < 0 ? 0 : (r > h - 1 ? h - 1 : r);
        acc = fma(taps[k], rp[r * cw + j], acc);
    }
    c32[i * pitch32 + j] = (float)acc;
    if (c64) c64[i * pitch64 + j] = acc;
}

// Reversed tap vector: entry k multiplies x[j - mr + k], i.e. h_N[mr - k].
void fill_taparg(const Taps &t, TapArg &a) {
    const int nt = t.ml + t.mr + 1;
    for (int k = 0; k < nt; k++) a.h[k] = t.h[t.mr - k + t.ml];
}

// Blocks per SM of one fused instantiation at its shared memory (cached per
// device); also raises the kernel's dynamic shared-memory limit.
template <typename P, int MT>
int fused_blocks_per_sm(int *bps) {
    static std::mutex mu;
    static std::map<int, int> done;
    int dev = 0;
    GPV_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    auto it = done.find(dev);
    if (it == done.end()) {
        constexpr size_t smem = Fused<P, MT>::kSmem;
        GPV_CUDA_TRY(cudaFuncSetAttribute(prefilter_fused<P, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int n = 0;
        GPV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, prefilter_fused<P, MT>, kFusedThreads, smem));
        it = done.emplace(dev, n > 0 ? n : 1).first;
    }
    *bps = it->second;
    return GPV_SUCCESS;
}

// Coefficient rows [lo, hi) of an image whose lines both have at least kT
// samples, lead-in MT; lo is a multiple of kQ, and hi too unless it is the last
// row's end (the groups of outputs are cut at multiples of kQ).  The rows are
// split into the number of segments that makes the last wave of blocks end
// first, each segment paying for its 2 MT lead-in lines: a 4096^2 image has
// blocks for several waves whatever the split, but a strip per 32 columns
// of a 1237-pixel-wide one leaves three quarters of the SMs idle unless its
// rows are cut short.
template <typename P, int MT>
int launch_fused(gpv_image *img, const P *px, cudaStream_t s, int64_t lo, int64_t hi) {
    if (hi <= lo) return GPV_SUCCESS;
    int bps = 1;
    if (int rc = fused_blocks_per_sm<P, MT>(&bps)) return rc;
    const int64_t strips = (img->cw + kStrip - 1) / kStrip, rows = hi - lo;
    const int64_t slots = (int64_t)bps * std::max(1, img->ctx->num_sms);
    int64_t seg = rows, best = INT64_MAX;
    for (int64_t n = 1; n <= (rows + kQ - 1) / kQ; n++) {
        const int64_t len = ((rows + n - 1) / n + kQ - 1) / kQ * kQ, k = (rows + len - 1) / len;
        const int64_t cost = (strips * k + slots - 1) / slots * (len + 2 * MT);
        if (cost < best) {
            best = cost;
            seg = len;
        }
    }
    const int64_t segs = (rows + seg - 1) / seg;
    static const Poles kPoles = poles();
    prefilter_fused<P, MT><<<dim3((unsigned)strips, (unsigned)segs), kFusedThreads, Fused<P, MT>::kSmem, s>>>(
        px, img->h, img->w, img->border, img->cw, img->ch, lo, hi, seg, kPoles, img->c32, img->pitch32, img->c64,
        img->pitch64);
    GPV_CUDA_TRY(cudaGetLastError());
    return GPV_SUCCESS;
}

template <typename P>
int launch_fused_rows(gpv_image *img, const P *px, cudaStream_t s, int64_t lo, int64_t hi) {
    // coefficients kept in FP32 only: |m| <= kM32
    return img->c64 == nullptr ? launch_fused<P, kM32>(img, px, s, lo, hi) : launch_fused<P, kM>(img, px, s, lo, hi);
}

bool long_lines(const gpv_image *img) { return img->cw >= kT && img->ch >= kT; }

template <typename P>
int run_prefilter(gpv_image *img, const P *px, cudaStream_t s) {
    if (long_lines(img)) return launch_fused_rows(img, px, s, 0, img->ch);
    const Taps &tr = taps_for(img->cw);
    const Taps &tc = taps_for(img->ch);
    // a short line: every circulant tap, through the FP64 row-pass buffer
    {
        const int nt = tr.ml + tr.mr + 1;
        TapArg a;
        fill_taparg(tr, a);
        double *dt = reinterpret_cast<double *>(img->rowpass) + img->h * img->cw;  // tap scratch after the row pass
        GPV_CUDA_TRY(cudaMemcpyAsync(dt, a.h, sizeof(double) * nt, cudaMemcpyHostToDevice, s));
        const int64_t total = img->h * img->cw;
        rowpass_small<P><<<(unsigned)((total + 255) / 256), 256, 0, s>>>(px, img->h, img->w, img->border, img->cw,
                                                                          tr.mr, nt, dt, img->rowpass);
        GPV_CUDA_TRY(cudaStreamSynchronize(s));  // host tap array is reused below
    }
    GPV_CUDA_TRY(cudaGetLastError());
    {
        const int nt = tc.ml + tc.mr + 1;
        TapArg a;
        fill_taparg(tc, a);
        double *dt = reinterpret_cast<double *>(img->rowpass) + img->h * img->cw + kT;
        GPV_CUDA_TRY(cudaMemcpyAsync(dt, a.h, sizeof(double) * nt, cudaMemcpyHostToDevice, s));
        const int64_t total = img->ch * img->cw;
        colpass_small<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(img->rowpass, img->h, img->cw, img->ch,
                                                                        img->border, tc.mr, nt, dt, img->c32,
                                                                        img->pitch32, img->c64, img->pitch64);
        GPV_CUDA_TRY(cudaStreamSynchronize(s));
    }
    GPV_CUDA_TRY(cudaGetLastError());
    return GPV_SUCCESS;
}

}  // namespace

const Taps &taps_for(int64_t n) {
    std::lock_guard<std::mutex> lk(g_taps_mu);
    auto it = g_taps.find(n);
    if (it != g_taps.end()) return it->second;
    Taps t;
    t.n = (int)n;
    if (n >= kT) {
        t.ml = t.mr = kM;
    } else {  // all n residues once: offsets -(n-1)/2 .. n/2
        t.ml = (int)((n - 1) / 2);
        t.mr = (int)(n / 2);
    }
    t.h.resize(t.ml + t.mr + 1);
    // spectrum of the zero-phase kernel (build_kernel) in closed form
    std::vector<double> inv(n);
    for (int64_t j = 0; j < n; j++) {
        const double wj = 2.0 * M_PI * (double)j / (double)n;
        inv[j] = 1.0 / (11.0 / 20.0 + (13.0 / 30.0) * std::cos(wj) + (1.0 / 60.0) * std::cos(2.0 * wj));
    }
    for (int m = -t.ml; m <= t.mr; m++) {
        // cos(2 pi j m / n) with the argument reduced exactly: (j*m) mod n
        double acc = 0.0;
        for (int64_t j = 0; j < n; j++) {
            int64_t q = ((j * (int64_t)m) % n + n) % n;
            acc += std::cos(2.0 * M_PI * (double)q / (double)n) * inv[j];
        }
        t.h[m + t.ml] = acc / (double)n;
    }
    return g_taps.emplace(n, std::move(t)).first->second;
}

namespace {
// Host pixels in row chunks into img->px_dev on the copy stream cs.  As each
// chunk lands, the groups of coefficient rows whose lines all come from rows
// already landed are filtered on s, so the copies overlap the filtering; the
// first groups (their lines wrap to the image's last rows) go after the last
// chunk.  Images with a short line take the whole copy, then
// the ordinary prefilter.
template <typename P>
int prefilter_host(gpv_image *img, const P *px_host, cudaStream_t s, cudaStream_t cs, cudaEvent_t *ev, int nev) {
    P *dst = static_cast<P *>(img->px_dev);
    const size_t row_bytes = sizeof(P) * (size_t)img->w;
    // rows per copy: ceil(h / (nev - 1)) rounded up to 32, so at most nev - 1
    // chunks (events ev[1 .. nev-1]) cover the image
    const int64_t chunk = ((img->h + nev - 2) / (nev - 1) + 31) / 32 * 32;
    // the copies wait for earlier work on s that may still read px_dev
    GPV_CUDA_TRY(cudaEventRecord(ev[0], s));
    GPV_CUDA_TRY(cudaStreamWaitEvent(cs, ev[0], 0));
    if (!long_lines(img) || img->h < 2 * 32 * (nev - 1)) {
        GPV_CUDA_TRY(cudaMemcpyAsync(dst, px_host, row_bytes * (size_t)img->h, cudaMemcpyHostToDevice, cs));
        GPV_CUDA_TRY(cudaEventRecord(ev[1], cs));
        GPV_CUDA_TRY(cudaStreamWaitEvent(s, ev[1], 0));
        return run_prefilter(img, static_cast<const P *>(dst), s);
    }
    const int64_t mt = img->c64 == nullptr ? kM32 : kM;
    // coefficient rows [0, first) wait for the last chunk (their lines wrap to the last rows)
    const int64_t first = (mt + kQ - 1) / kQ * kQ;
    int64_t lo = first;
    int k = 1;
    for (int64_t r0 = 0; r0 < img->h; r0 += chunk, k++) {
        // the last event takes whatever rows remain (never an event past ev[nev - 1])
        const int64_t nr = k == nev - 1 ? img->h - r0 : std::min(chunk, img->h - r0);
        GPV_CUDA_TRY(cudaMemcpyAsync(dst + r0 * img->w, px_host + r0 * img->w, row_bytes * (size_t)nr,
                                     cudaMemcpyHostToDevice, cs));
        GPV_CUDA_TRY(cudaEventRecord(ev[k], cs));
        GPV_CUDA_TRY(cudaStreamWaitEvent(s, ev[k], 0));
        // a group of coefficient rows ending at i reads image rows below min(h, i + mt - border)
        const int64_t landed = r0 + nr;
        const int64_t hi = landed >= img->h ? img->ch : (landed - mt + img->border) / kQ * kQ;
        if (hi > lo) {
            if (int rc = launch_fused_rows(img, static_cast<const P *>(dst), s, lo, hi)) return rc;
            lo = hi;
        }
    }
    return launch_fused_rows(img, static_cast<const P *>(dst), s, 0, first);
}
}  // namespace

int prefilter_from_host(gpv_image *img, const void *px_host, int dtype, cudaStream_t s, cudaStream_t cs,
                        cudaEvent_t *ev, int nev) {
    switch (dtype) {
        case GPV_U8: return prefilter_host(img, static_cast<const uint8_t *>(px_host), s, cs, ev, nev);
        case GPV_U16: return prefilter_host(img, static_cast<const uint16_t *>(px_host), s, cs, ev, nev);
        case GPV_F32: return prefilter_host(img, static_cast<const float *>(px_host), s, cs, ev, nev);
        case GPV_F64: return prefilter_host(img, static_cast<const double *>(px_host), s, cs, ev, nev);
        default: set_error("unknown pixel dtype"); return GPV_ERR_INVALID;
    }
}

size_t prefilter_rowpass_bytes(int64_t h, int64_t cw, int64_t ch) {
    // the row pass plus two tap vectors of scratch, for the short-line kernels only
    return (cw >= kT && ch >= kT) ? 0 : sizeof(double) * (size_t)(h * cw + 2 * kT + 8);
}

int prefilter_launch(gpv_image *img, const void *px_dev, int dtype, cudaStream_t s) {
    switch (dtype) {
        case GPV_U8: return run_prefilter(img, static_cast<const uint8_t *>(px_dev), s);
        case GPV_U16: return run_prefilter(img, static_cast<const uint16_t *>(px_dev), s);
        case GPV_F32: return run_prefilter(img, static_cast<const float *>(px_dev), s);
        case GPV_F64: return run_prefilter(img, static_cast<const double *>(px_dev), s);
        default: set_error("unknown pixel dtype"); return GPV_ERR_INVALID;
    }
}

}  // namespace gpv
