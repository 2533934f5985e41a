// icgn_runs.cu -- mixed-precision ICGN with the circular template cut into
// vertical runs: one thread block per subset at a time, the subset's
// coefficient windows staged in shared memory, and every lane walking runs
// of K vertically adjacent template pixels with the 6 x 6 coefficient block
// of the current sample held in registers.
//
// Same algorithm and numerics contract as the other solve kernels --
// Subset::new + solve_icgn_result, src/subset.rs:836-919, 1117-1219 -- laid
// out for the B200's issue and shared-memory rates:
//  * Template runs.  The square around the circle (src/masks.rs:69-109) is
//    cut into bands of K rows; a band's columns dx in [-w, w] (w: the widest
//    circle row of the band) are its tasks, each task the K pixels
//    (dx, dy0 .. dy0 + K - 1) with a bit per pixel for the circle (and the
//    global mask).  The last band is moved up to end at dy = r, its rows
//    already covered above masked off.  Tasks are dealt to threads in band
//    order, so a warp's lanes hold neighbouring columns of one band.
//  * Sample loop.  Vertically adjacent template pixels land one coefficient
//    row apart after any warp of moderate strain, so a lane keeps the 6 x 6
//    coefficients of its last sample in registers and, when the next
//    sample's block is the same one moved down a row (same column, next
//    row), loads only the new row: 6 shared-memory loads per sample instead
//    of 36.  A sample whose block moved otherwise reloads all six rows (a
//    divergent branch taken by few lanes).  The taps and the row combine run
//    as sm_100 paired FP32 ops on symmetric weight pairs (b_k, b_{5-k}).
//  * Setup.  Every template pixel of an interior subset sits at an integer
//    offset from the centre, so f's value and gradient rows share one basis:
//    each run forms its K + 5 coefficient-row sums once (paired FMAs over
//    row pairs) and combines six of them per pixel.  The Hessian's gradient
//    moments are accumulated per run as powers of dy and expanded by powers
//    of the run's dx once per run.
//  * Hessian.  Factored once per subset (Cholesky of the Jacobi-scaled
//    matrix, FP64, one warp), and its inverse formed from the factor
//    (H^-1 = D L^-T L^-1 D); each iteration's increment is that inverse times
//    the gradient (FP64, 12 lanes).
//  * Instruction fetch.  An SM caches 32 KB of instructions (8 KB next to each
//    scheduler); past that they come from a cache that several SMs share, and
//    that cache was 81 % busy: the solve's blocks walk some 100 KB of code, each
//    in its own phase.  So the stretches run once or a few times per subset
//    are kept short -- the factor as passes of rolled loops, the sums over lanes
//    through shared memory instead of unrolled shuffles, the omitted-mode
//    diagnostic only in the kernels of launches that ask for it.  Measured with
//    the loads of records past L1 (they are read once per iteration) and the
//    floors by rounding: 37-40k second-order subsets of radius 30 / 24 / 16
//    5.71 -> 5.36, 4.80 -> 4.23, 3.99 -> 3.24 ms, 27k first-order ones of
//    radius 25 2.35 -> 2.18 ms; the shared cache 67 % busy.  A pool of 16 warps per
//    SM sharing five subsets (no block barriers) measured 2.6 times slower: its
//    warps fetch each stretch alone, at 93 % of that cache.
//  * Sums.  The per-iteration sums g - f_m, its square and (f - f_m)(g - f_m)
//    are FP32 over one run (at most K samples), then FP64 per thread and across
//    the block in a fixed order (deterministic); the steepest-descent products
//    and the setup's sums are FP32 per thread, then FP64.  64 threads keep
//    the FP32 sums of 128: two apiece, one after the other.
//  * Rigid texture (RIGID; orders 1 and 2): the grain maps sampled per pixel at
//    setup, and a template pass per iteration with the sums of its correction G
//    (the run's four pixels' loads together in flight); the sample loop only adds
//    G to its cross term.  14,420 second-order subsets of radius 30 4.33 ms in the
//    tiled kernel, 3.2 here (deformable 2.0).  With the diagnostic the tiled
//    kernel stays: see the launcher.
// Subsets whose warped square leaves the image or the staged window take a
// clamped per-sample path (the reference's edge clamp, src/image.rs:129-132),
// reading the window with clamped indices or global memory.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <map>
#include <mutex>
#include <utility>

#include "icgn_runs.cuh"

namespace gpv {
namespace {

constexpr int kBufPitch = 9;  // a warp's staging of sums over lanes: 32 rows of 8 values

// NW: warps per block (block sums are kept per warp)
template <int NW>
struct RunSmem {
    double mom[3 * 15];
    double L[144];     // the Cholesky factor's inverse (row-major)
    double Hi[160];    // the factor's columns, then H^-1
    float part[NW][32 * kBufPitch];  // per-warp staging of the sums over lanes
    double linv[12];   // 1 / L_jj
    double dsc[12];    // Jacobi scale 1 / sqrt(H_jj)
    double A[12], S[12];
    double p[12], pprev[12], dp[12], grad[12];
    double red[NW][16];
    double red2[NW][80];
    double aug[80];
    double misc[10];
    int flag[4];
    int item;
    int n_valid;
    int win_r0, win_c0, win_h, win_w, win_p, win_ok;
};

// Plan g's or f's window over pixels [xlo, xhi] x [ylo, yhi] and stage it in
// win by threads [t0, NT): 16-byte asynchronous global-to-shared copies
// (cp.async, no registers held for the data), so all of a thread's copies
// are in flight at once; rows and columns outside the coefficients are
// clamped.  Each thread waits for its own copies before it returns, and the
// caller's block barrier publishes the window and its place in sm (win_ok:
// it fits and is staged).  Both addresses are 16-byte aligned: coefficient rows
// are a multiple of 32 floats apart, c0 and the clamped columns are multiples
// of 4, and the window's pitch is a multiple of 4 floats (run_pitch).
template <int NT>
__device__ __forceinline__ void place_window(RunSmem<NT / 32> &sm, const float *__restrict__ C, int64_t cpitch, int ch,
                                             int border, int cap, int xlo, int xhi, int ylo, int yhi, float *win, int t0) {
    int r0, c0, wh, ww, pitch;
    const bool ok = run_plan<32>(xlo, xhi, ylo, yhi, border, cap, r0, c0, wh, ww, pitch);
    if (ok) {
        const int nv = ww >> 2;
#pragma unroll 2
        for (int idx = (int)threadIdx.x - t0; idx < wh * nv; idx += NT - t0) {
            const int rr = idx / nv, cc = (idx - rr * nv) << 2;
            const int row = max(min(r0 + rr, ch - 1), 0), col = max(min(c0 + cc, (int)cpitch - 4), 0);
            const unsigned dst = (unsigned)__cvta_generic_to_shared(win + rr * pitch + cc);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(C + (int64_t)row * cpitch + col)
                         : "memory");
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    }
    if ((int)threadIdx.x == t0) {
        sm.win_ok = ok;
        sm.win_r0 = r0; sm.win_c0 = c0; sm.win_h = wh; sm.win_w = ww; sm.win_p = pitch;
    }
}

// Sums over a warp's lanes (FP64) of up to 8 columns of its staging buffer
// (32 rows, pitch 9: no bank conflicts either way) into dst[0 .. g): eight
// lanes per quarter of the rows, two chains a lane.
__device__ __forceinline__ void column_sums(const float *buf, double *dst, int g, int lane) {
    const float *p = buf + (lane >> 3) * (8 * kBufPitch) + (lane & 7);
    double s0 = (double)p[0], s1 = (double)p[kBufPitch];
#pragma unroll
    for (int i = 2; i < 8; i += 2) {
        s0 += (double)p[i * kBufPitch];
        s1 += (double)p[(i + 1) * kBufPitch];
    }
    s0 += s1;
    s0 += __shfl_xor_sync(0xffffffffu, s0, 8);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 16);
    if (lane < g) dst[lane] = s0;
}

// Warp sums (FP64) of N FP32 values per lane into dst[0..N) through the
// warp's staging buffer, 8 at a time.  A butterfly of shuffles per 16 values
// took 2.4 times the instructions (64-bit shuffles are two each).  ROLLED: the
// values pass through local memory so that the groups are passes of one
// loop: the setup's 73 values would otherwise unroll to ten copies.
template <int N, bool ROLLED>
__device__ __forceinline__ void run_warp_sums(const float (&a)[N], float *buf, double *dst, int lane) {
    if constexpr (ROLLED) {
        constexpr int G = (N + 7) / 8;
        float v[G * 8];
#pragma unroll
        for (int q = 0; q < G * 8; q++) v[q] = q < N ? a[q] : 0.f;
#pragma unroll 1
        for (int g = 0; g < G; g++) {
            __syncwarp();  // the buffer's last reader is done
#pragma unroll
            for (int j = 0; j < 8; j++) buf[lane * kBufPitch + j] = v[g * 8 + j];
            __syncwarp();
            column_sums(buf, dst + g * 8, min(8, N - g * 8), lane);
        }
    } else {
#pragma unroll
        for (int g = 0; g < N; g += 8) {
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8 && g + j < N; j++) buf[lane * kBufPitch + j] = a[g + j];
            __syncwarp();
            column_sums(buf, dst + g, min(8, N - g), lane);
        }
    }
}

// 1.5 x 2^23: adding it rounds an FP32 value of magnitude below 2^22 to an
// integer, which then stands in the sum's low mantissa bits (offset by kMagic's
// own bits, the bias that the window offsets take off again).
constexpr float kMagic = 12582912.0f;
constexpr uint32_t kMagicBits = 0x4B400000u;

// The quintic basis at u = fraction - 1/2 as symmetric pairs W[k] = (w_k,
// w_{5-k}), k = 0..2: the weights of basis() split into an even part
// e_k(v) and an odd part -u q_k(v), v = u^2, w_k = e_k - u q_k and
// w_{5-k} = e_k + u q_k, each one FMA (the odd part is never rounded on its
// own), in scalar FP32 ops whose polynomial coefficients are instruction
// immediates (as paired ops the coefficients take 18 registers, which the
// sample loop does not have: 53 M sectors of spills on 8,836 second-order
// subsets, 1.46 against 1.33 ms).
__device__ __forceinline__ void basis_sym(float u, float2 W[3]) {
    const float v = u * u;
    const float e0 = fmaf(fmaf(v, 1.0f / 48.0f, 1.0f / 96.0f), v, 1.0f / 3840.0f);
    const float e1 = fmaf(fmaf(v, -1.0f / 16.0f, 7.0f / 32.0f), v, 79.0f / 1280.0f);
    const float e2 = fmaf(fmaf(v, 1.0f / 24.0f, -11.0f / 48.0f), v, 841.0f / 1920.0f);
    const float q0 = fmaf(fmaf(v, 1.0f / 120.0f, 1.0f / 48.0f), v, 1.0f / 384.0f);
    const float q1 = fmaf(fmaf(v, -1.0f / 24.0f, 1.0f / 16.0f), v, 25.0f / 128.0f);
    const float q2 = fmaf(fmaf(v, 1.0f / 12.0f, -7.0f / 24.0f), v, 77.0f / 192.0f);
    W[0] = make_float2(fmaf(-u, q0, e0), fmaf(u, q0, e0));
    W[1] = make_float2(fmaf(-u, q1, e1), fmaf(u, q1, e1));
    W[2] = make_float2(fmaf(-u, q2, e2), fmaf(u, q2, e2));
}

// A record, read once per iteration: not kept in L1.
__device__ __forceinline__ float4 ld_rec(const float4 *p) {
    float4 v;
    asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ float ld_once(const float *p) {
    float v;
    asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// One coefficient row against the column weights: sum_k b_k c_k with the
// pairs (c_k, c_{5-k}) x (b_k, b_{5-k}).
__device__ __forceinline__ float row_dot(const float (&c)[6], const float2 B[3]) {
    float2 s = __fmul2_rn(make_float2(c[0], c[5]), B[0]);
    s = __ffma2_rn(make_float2(c[1], c[4]), B[1], s);
    s = __ffma2_rn(make_float2(c[2], c[3]), B[2], s);
    return s.x + s.y;
}

__device__ __forceinline__ float combine6(const float (&s)[6], const float2 A[3]) {
    float2 v = __fmul2_rn(make_float2(s[0], s[5]), A[0]);
    v = __ffma2_rn(make_float2(s[1], s[4]), A[1], v);
    v = __ffma2_rn(make_float2(s[2], s[3]), A[2], v);
    return v.x + v.y;
}

// Per-run FP32 accumulators of the iteration sums.
struct RunAcc {
    float p1, p2, pfg;
    float2 m0, m1, m2;  // sum G, sum G dy, sum G dy^2 with G = (gx, gy) (g - f_m)
};

// A Kahan-compensated FP64 sum: add() carries the rounding error of each
// addition into the next one.
struct KSum {
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add(double x) {
        const double y = x - c, t = s + y;
        c = (t - s) - y;
        s = t;
    }
};

// One sample: rec = (df/dx, df/dy, f - s, w) with w = 1 for template
// pixels, 0 outside (the gradient pair first: one aligned register pair,
// so the steepest-descent products and sums are paired FP32 operations);
// pfg sums (f - s)(g - f_m) (corrected to f - f_m with the block totals).  KAHAN: the three ZNSSD sums (g - f_m, its square and
// the cross term) go straight into the thread's compensated FP64 sums ks
// instead of the run's FP32 partials.
template <int ORDER, bool KAHAN>
__device__ __forceinline__ void acc_sample(RunAcc &a, KSum (&ks)[3], float4 rec, float g, float fmf, float2 dy2, float2 dd2) {
    const float gc = (g - fmf) * rec.w;
    if (KAHAN) {
        const double gd = (double)gc;
        ks[0].add(gd);
        ks[1].add(gd * gd);
        ks[2].add((double)rec.z * gd);
    } else {
        a.p1 += gc;
        a.p2 = fmaf(gc, gc, a.p2);
        a.pfg = fmaf(rec.z, gc, a.pfg);
    }
    const float2 gxy = __fmul2_rn(make_float2(rec.x, rec.y), make_float2(gc, gc));
    a.m0 = __fadd2_rn(a.m0, gxy);
    if (ORDER >= 1) a.m1 = __ffma2_rn(gxy, dy2, a.m1);
    if (ORDER == 2) a.m2 = __ffma2_rn(gxy, dd2, a.m2);
}

// The run's steepest-descent sums into the thread's totals PB[mu] (pairs
// (gx, gy) of monomial mu = 1, dx, dy, dx^2/2, dx dy, dy^2/2).
template <int ORDER>
__device__ __forceinline__ void acc_expand(const RunAcc &a, float dxf, float2 (&PB)[6]) {
    PB[0] = __fadd2_rn(PB[0], a.m0);
    if (ORDER >= 1) {
        PB[1] = __ffma2_rn(make_float2(dxf, dxf), a.m0, PB[1]);
        PB[2] = __fadd2_rn(PB[2], a.m1);
    }
    if (ORDER == 2) {
        const float h = 0.5f * dxf * dxf;
        PB[3] = __ffma2_rn(make_float2(h, h), a.m0, PB[3]);
        PB[4] = __ffma2_rn(make_float2(dxf, dxf), a.m1, PB[4]);
        PB[5] = __ffma2_rn(make_float2(0.5f, 0.5f), a.m2, PB[5]);
    }
}

// Omitted-mode diagnostic at the last sampled warp: g sampled again into RSG
// (the solve keeps no samples), then eta_two_pass.  Only kernels instantiated
// for it hold it: inside every solve it cost 4 % in registers and code.
// fms: s - f_m.
template <int ORDER, int NT, int K>
__device__ __forceinline__ void run_eta(RunSmem<NT / 32> &sm, const float *win, const float *__restrict__ g32, int64_t pitch32,
                                     int w, int h, int B, const int2 *tasks, int T, const float4 *REC, float *RSG,
                                     const int *RVM, double cx, double cy, double fms, double dn, double df, double gm,
                                     double dg, double *eu, double *ev) {
    constexpr int M = Ord<ORDER>::M;
    const int tid = threadIdx.x;
    const double *pprev = sm.pprev;
    const double X0 = cx + pprev[0], Y0 = cy + pprev[1];
    const double bxd = floor(X0), byd = floor(Y0);
    const int wbx = (int)bxd, wby = (int)byd;
    const double ox = X0 - bxd, oy = Y0 - byd;
    const bool staged = sm.win_ok != 0;  // the window the last iteration sampled
    const int gr0 = sm.win_r0, gc0 = sm.win_c0, gwh = sm.win_h, gww = sm.win_w, gP = sm.win_p;
    // this thread's template pixels; the first walk samples g again
    auto each = [&](auto first, auto fn) {
#pragma unroll 1
        for (int t = tid; t < T; t += NT) {
            int dxi, dy0;
            unpack_task(tasks[t], dxi, dy0);
            const int vm = RVM[t];
#pragma unroll 1
            for (int j = 0; j < K; j++) {
                if (!((vm >> j) & 1)) continue;
                const int sl = j * T + t;
                const double dx = dxi, dy = dy0 + j;
                if constexpr (decltype(first)::value) {
                    double lx = ox + dx, ly = oy + dy;
                    if (ORDER >= 1) {
                        lx += pprev[2] * dx + pprev[4] * dy;
                        ly += pprev[3] * dx + pprev[5] * dy;
                    }
                    if (ORDER == 2) {
                        lx += 0.5 * pprev[6 % M] * dx * dx + pprev[8 % M] * dx * dy + 0.5 * pprev[10 % M] * dy * dy;
                        ly += 0.5 * pprev[7 % M] * dx * dx + pprev[9 % M] * dx * dy + 0.5 * pprev[11 % M] * dy * dy;
                    }
                    int ix, iy;
                    float tx, ty;  // integer offsets added exactly, the small parts in FP32
                    split_clamped(wbx + dxi, (float)(lx - dx), w, ix, tx);
                    split_clamped(wby + dy0 + j, (float)(ly - dy), h, iy, ty);
                    float a[6], b[6];
                    basis(ty, a);
                    basis(tx, b);
                    if (staged) {
                        const int wx = min(max(ix + B - 2 - gc0, 0), gww - 6), wy = min(max(iy + B - 2 - gr0, 0), gwh - 6);
                        RSG[sl] = contract<float>(win + wy * gP + wx, gP, a, b);
                    } else {
                        RSG[sl] = contract<float>(g32 + (int64_t)(iy + B - 2) * pitch32 + (ix + B - 2), pitch32, a, b);
                    }
                }
                const float4 rec = REC[sl];
                fn((double)rec.z + fms, (double)rec.x, (double)rec.y, (double)RSG[sl] - gm, dx, dy);
            }
        }
    };
    auto red = [&](auto &v) { run_block_sums<NT>(v, sm.red2, sm.aug); };
    double u, v;
    eta_two_pass<ORDER>(dn, df, dg, each, red, u, v);
    *eu = u;
    *ev = v;
}

template <int ORDER, int NT, int K, bool KAHAN, bool ETA, bool RIGID>
__device__ void run_subset(const RunArgs &R, int idx, const gpv_subset_desc &d, float *base, float *win,
                           RunSmem<NT / 32> &sm) {
    const KArgs &A = R.k;
    using O = Ord<ORDER>;
    constexpr int M = O::M, NMU = O::NMU, NMOM = O::NMOM, NB = 2 * O::DEG + 1;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int r = d.radius;
    const int re = max(r, K - 1 - r);  // half side of the square the runs cover
    const int T = R.task_n[r];
    const int2 *tasks = R.tasks + R.task_off[r];
    // per-pixel records (df/dx, df/dy, f - s, 1 in the template / 0 outside:
    // zero gradients outside) in slot j * T + t of run t; eta resamples; run bits
    float4 *REC = reinterpret_cast<float4 *>(base);
    float *RSG = base + 4 * R.nslot;
    int *RVM = reinterpret_cast<int *>(base + 5 * R.nslot);
    // rigid texture: the grain maps at the pixels (three arrays), the template's
    // correction G of the iteration
    float *RH = base + run_plain_floats(R.nslot), *RTG = RH + 3 * R.nslot;
    const bool rigid_on = RIGID && A.grain_scal[4] != 0.0;  // uniform: the image has measurable speckle
    const double cx = d.coord[0], cy = d.coord[1];
    const int cxi = (int)cx, cyi = (int)cy;
    const double fxd = floor(cx), fyd = floor(cy);
    const int bx = (int)fxd, by = (int)fyd;
    const float fx = (float)(cx - fxd), fy = (float)(cy - fyd);
    const int B = A.border, ch = A.h + 2 * B;

    // ---- stage f's window ------------------------------------------------
    {
        // +-1: an FP32 fraction can round up to the next integer
        const int xlo = max(0, min(bx - re - 1, A.w - 1)), xhi = max(0, min(bx + re + 1, A.w - 1));
        const int ylo = max(0, min(by - re - 1, A.h - 1)), yhi = max(0, min(by + re + 1, A.h - 1));
        place_window<NT>(sm, A.f32, A.pitch32, ch, B, R.win_cap, xlo, xhi, ylo, yhi, win, 0);
        if (tid < M) {
            sm.p[tid] = d.p0[tid];
            sm.pprev[tid] = d.p0[tid];
        }
        __syncthreads();
    }
    const bool f_staged = sm.win_ok != 0;
    const int fr0 = sm.win_r0, fc0 = sm.win_c0, fwh = sm.win_h, fww = sm.win_w, fP = sm.win_p;
    // interior: every run pixel sits at an integer offset from the centre
    // inside the image, so all share one fraction and one basis
    const bool interior = f_staged && bx - re >= 0 && bx + re <= A.w - 1 && by - re >= 0 && by + re <= A.h - 1;

    // ---- setup, pass 1: f and its gradient per pixel, first sums ------------
    // [count, sum (f-s), sum (f-s)^2, SSSIG, Bf_j = sum SDI_j (f-s) (M),
    //  S_j = sum SDI_j (M)] about a subset-uniform level s (the coefficient
    // under the centre: keeps the sums free of cancellation and a flat
    // subset's sums exactly zero); FP32 per thread, FP64 across the block.
    constexpr int NVA = 4 + 2 * M;
    // 64 threads have twice the runs each: thread i takes the runs of threads i
    // and i + 64 of 128 one after the other, in FP32 sums of their own joined in
    // FP64, so that every FP32 sum is one that 128 threads have (the error of
    // delta_f and of the ZNCC against 64 bits would be 1.2 to 1.9 times as large)
    constexpr int kHalves = NT == 64 ? 2 : 1;
    double carry = 0.0;
    float acc[NVA];
    float shift;
    if (f_staged) {
        const int wx = min(max(max(0, min(bx, A.w - 1)) + B - fc0, 0), fww - 1);
        const int wy = min(max(max(0, min(by, A.h - 1)) + B - fr0, 0), fwh - 1);
        shift = win[wy * fP + wx];
    } else {
        shift = A.f32[(int64_t)(max(0, min(by, A.h - 1)) + B) * A.pitch32 + max(0, min(bx, A.w - 1)) + B];
    }
    auto pix1 = [&](bool v, float f, float gx, float gy, int dx, int dy) {
        if (!v) return;
        const float dxf = (float)dx, dyf = (float)dy;
        const float fs = f - shift;
        acc[0] += 1.f;
        acc[1] += fs;
        acc[2] = fmaf(fs, fs, acc[2]);
        acc[3] = fmaf(0.5f * gx, gx, fmaf(0.5f * gy, gy, acc[3]));
        const float gxf = gx * fs, gyf = gy * fs;
#pragma unroll
        for (int mu = 0; mu < NMU; mu++) {
            const float mv = mu_val<float>(mu, dxf, dyf);
            acc[4 + 2 * mu] = fmaf(gxf, mv, acc[4 + 2 * mu]);
            acc[5 + 2 * mu] = fmaf(gyf, mv, acc[5 + 2 * mu]);
            acc[4 + M + 2 * mu] = fmaf(gx, mv, acc[4 + M + 2 * mu]);
            acc[5 + M + 2 * mu] = fmaf(gy, mv, acc[5 + M + 2 * mu]);
        }
    };
    {
        float a0[6], da0[6], b0[6], db0[6];
        basis(fy, a0); dbasis(fy, da0);
        basis(fx, b0); dbasis(fx, db0);
        float2 bb[6], dbb[6];  // column weights as duplicated pairs (two rows per paired FMA)
#pragma unroll
        for (int k = 0; k < 6; k++) {
            bb[k] = make_float2(b0[k], b0[k]);
            dbb[k] = make_float2(db0[k], db0[k]);
        }
#pragma unroll 1
        for (int hf = 0; hf < kHalves; hf++) {
#pragma unroll
        for (int q = 0; q < NVA; q++) acc[q] = 0.f;
        for (int t = hf * NT + tid; t < T; t += kHalves * NT) {
            int dx, dy0;
            unpack_task(tasks[t], dx, dy0);
            uint32_t vm = (uint32_t)tasks[t].y;
            if (A.mask) {
#pragma unroll
                for (int j = 0; j < K; j++)
                    if (!mask_ok(A, cxi, cyi, dx, dy0 + j)) vm &= ~(1u << j);
            }
            RVM[t] = (int)vm;
            if (interior) {
                // coefficient-row sums (value and x-derivative weights) of the
                // run's K + 5 rows, two rows per paired FMA; then six rows per pixel
                const float *p0 = win + (by + dy0 + B - 2 - fr0) * fP + (bx + dx + B - 2 - fc0);
                float s[K + 6], q[K + 6];
#pragma unroll
                for (int m = 0; m + 1 < K + 5; m += 2) {
                    const float *r0 = p0 + m * fP, *r1 = r0 + fP;
                    float2 c = make_float2(r0[0], r1[0]);
                    float2 S2 = __fmul2_rn(c, bb[0]), D2 = __fmul2_rn(c, dbb[0]);
#pragma unroll
                    for (int k = 1; k < 6; k++) {
                        c = make_float2(r0[k], r1[k]);
                        S2 = __ffma2_rn(c, bb[k], S2);
                        D2 = __ffma2_rn(c, dbb[k], D2);
                    }
                    s[m] = S2.x; s[m + 1] = S2.y;
                    q[m] = D2.x; q[m + 1] = D2.y;
                }
                if ((K + 5) & 1) {  // the last row alone (no row past the window)
                    const float *r0 = p0 + (K + 4) * fP;
                    float sv = r0[0] * b0[0], qv = r0[0] * db0[0];
#pragma unroll
                    for (int k = 1; k < 6; k++) {
                        sv = fmaf(r0[k], b0[k], sv);
                        qv = fmaf(r0[k], db0[k], qv);
                    }
                    s[K + 4] = sv;
                    q[K + 4] = qv;
                }
#pragma unroll
                for (int j = 0; j < K; j++) {
                    float val = 0.f, vx = 0.f, vy = 0.f;
#pragma unroll
                    for (int rr = 0; rr < 6; rr++) {
                        val = fmaf(a0[rr], s[j + rr], val);
                        vx = fmaf(a0[rr], q[j + rr], vx);
                        vy = fmaf(da0[rr], s[j + rr], vy);
                    }
                    const bool v = (vm >> j) & 1u;
                    REC[j * T + t] = v ? make_float4(vx, vy, val - shift, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
                    pix1(v, val, vx, vy, dx, dy0 + j);
                }
            } else {
#pragma unroll 1
                for (int j = 0; j < K; j++) {
                    const bool v = (vm >> j) & 1u;
                    int ix, iy;
                    float tx, ty;
                    split_clamped(bx, fx + (float)dx, A.w, ix, tx);
                    split_clamped(by, fy + (float)(dy0 + j), A.h, iy, ty);
                    float a[6], da[6], b[6], db[6];
                    basis(ty, a); dbasis(ty, da);
                    basis(tx, b); dbasis(tx, db);
                    float f, gx, gy;
                    if (f_staged) {
                        const int wx = min(max(ix + B - 2 - fc0, 0), fww - 6), wy = min(max(iy + B - 2 - fr0, 0), fwh - 6);
                        f = contract_grad<float>(win + wy * fP + wx, fP, a, da, b, db, gx, gy);
                    } else {
                        const float *F = A.f32 + (int64_t)(iy + B - 2) * A.pitch32 + (ix + B - 2);
                        f = contract_grad<float>(F, A.pitch32, a, da, b, db, gx, gy);
                    }
                    REC[j * T + t] = v ? make_float4(gx, gy, f - shift, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
                    pix1(v, f, gx, gy, dx, dy0 + j);
                }
            }
        }
        run_warp_sums<NVA, (NVA > 16)>(acc, sm.part[wid], sm.red2[wid], lane);
        if constexpr (kHalves == 2) {
            static_assert(NVA <= 32, "one sum per lane");
            __syncwarp();
            if (lane < NVA) {
                carry += sm.red2[wid][lane];
                sm.red2[wid][lane] = carry;
            }
            __syncwarp();
        }
        }
    }
    // ---- setup, pass 2: the Hessian's gradient moments ----------------------
    // sum g_p g_q dx^a dy^b (a + b <= 2 DEG) per run as powers of dy, then
    // expanded by the run's powers of dx; each thread re-reads its own records
    {
        float mom[3 * NMOM];
        double carry_m[(3 * NMOM + 31) / 32] = {};
#pragma unroll 1
        for (int hf = 0; hf < kHalves; hf++) {
#pragma unroll
        for (int q = 0; q < 3 * NMOM; q++) mom[q] = 0.f;
        for (int t = hf * NT + tid; t < T; t += kHalves * NT) {
            int dx, dy0;
            unpack_task(tasks[t], dx, dy0);
            float V[3][NB];
#pragma unroll
            for (int p = 0; p < 3; p++)
#pragma unroll
                for (int b = 0; b < NB; b++) V[p][b] = 0.f;
#pragma unroll
            for (int j = 0; j < K; j++) {
                const float4 rec = REC[j * T + t];
                const float gx = rec.x, gy = rec.y;  // zero for pixels outside the template
                const float gg[3] = {gx * gx, gx * gy, gy * gy};
                const float dyf = (float)(dy0 + j);
                float pw = 1.f;
#pragma unroll
                for (int b = 0; b < NB; b++) {
#pragma unroll
                    for (int p = 0; p < 3; p++) V[p][b] = fmaf(gg[p], pw, V[p][b]);
                    pw *= dyf;
                }
            }
            const float dxf = (float)dx;
            float xp[NB];
            xp[0] = 1.f;
#pragma unroll
            for (int a = 1; a < NB; a++) xp[a] = xp[a - 1] * dxf;
#pragma unroll
            for (int a = 0; a < NB; a++)
#pragma unroll
                for (int b = 0; a + b < NB; b++)
#pragma unroll
                    for (int p = 0; p < 3; p++)
                        mom[p * NMOM + mom_idx(a, b)] = fmaf(xp[a], V[p][b], mom[p * NMOM + mom_idx(a, b)]);
        }
        run_warp_sums<3 * NMOM, (NMOM > 1)>(mom, sm.part[wid], sm.red2[wid] + NVA, lane);
        if constexpr (kHalves == 2) {
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 3 * NMOM; q += 32) {
                if (q + lane < 3 * NMOM) {
                    carry_m[q / 32] += sm.red2[wid][NVA + q + lane];
                    sm.red2[wid][NVA + q + lane] = carry_m[q / 32];
                }
            }
            __syncwarp();
        }
        }
    }
    if constexpr (RIGID) {
        if (rigid_on) {
#pragma unroll 1
            for (int t = tid; t < T; t += NT) {
                int dx, dy0;
                unpack_task(tasks[t], dx, dy0);
#pragma unroll 1
                for (int j = 0; j < K; j++) {
                    float hv[3];
                    grain_sample(A.grain, A.h, A.w, cx + (double)dx, cy + (double)(dy0 + j), hv);
#pragma unroll
                    for (int m = 0; m < 3; m++) RH[m * R.nslot + j * T + t] = hv[m];
                }
            }
        }
    }
    __syncthreads();
    constexpr int NV = NVA + 3 * NMOM;
    if (wid == 0) {
        // block sums of the warp partials, then f_m, delta_f, A_j, S_j, the
        // Hessian and its factor (warp 0) while the other warps stage g's window
        for (int q = lane; q < NV; q += 32) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < NT / 32; w++) t += sm.red2[w][q];
            sm.aug[q] = t;
        }
        __syncwarp();
        const int n = (int)(sm.aug[0] + 0.5);
        const double dn = (double)n, ms = sm.aug[1] / (n > 0 ? dn : 1.0);  // mean of f - s
        const double fm = (double)shift + ms;
        const double saa = sm.aug[2] - ms * sm.aug[1];  // sum (f - f_m)^2
        int st = GPV_OK;
        if (n == 0) st = GPV_EMPTY_MASK;
        else if (!(sqrt(fmax(saa, 0.0) / dn) > 1e-6 * fmax(1.0, fabs(fm)))) st = GPV_FEATURELESS;  // flat subset
        if (st == GPV_OK) {
            if (lane < M) {
                sm.A[lane] = sm.aug[4 + lane] - ms * sm.aug[4 + M + lane];  // sum SDI (f - f_m)
                sm.S[lane] = sm.aug[4 + M + lane];
            }
            if (lane < 3 * NMOM) sm.mom[lane] = sm.aug[NVA + lane];
            if (lane + 32 < 3 * NMOM) sm.mom[lane + 32] = sm.aug[NVA + lane + 32];
            __syncwarp();
            if (!hess_factor<ORDER>(sm.mom, sm.Hi, sm.L, sm.linv, sm.dsc, lane)) st = GPV_SINGULAR_H;
        }
        if (lane == 0) {
            sm.flag[0] = st;
            sm.misc[5] = fm;
            sm.misc[6] = saa;
            sm.misc[7] = sm.aug[3];
            sm.n_valid = n;
        }
    } else {
        // stage g's window around the initial warp
        const int4 ext = run_extent<ORDER>(sm.p, cx, cy, re, A.w, A.h);
        place_window<NT>(sm, A.g32, A.pitch32, ch, B, R.win_cap, ext.x & ~kInside, ext.y, ext.z, ext.w, win, 32);
    }
    __syncthreads();
    const int st0 = sm.flag[0];
    const int n = sm.n_valid;
    const double dn = (double)n;
    const double fm = sm.misc[5], saa = sm.misc[6], tot_sssig = sm.misc[7];
    const float fmf = (float)fm;
    const double df = sqrt(fmax(saa, 0.0));
    if (st0 != GPV_OK) {
        if (tid == 0) {
            write_failed(A, idx, d, M, st0, n, n ? fm : 0.0, n ? df : 0.0);
            if (st0 == GPV_SINGULAR_H) {
                A.out[idx].sssig = tot_sssig;
                A.out[idx].sigma = sqrt(saa / dn);
            }
        }
        return;
    }
    // H^-1 by every thread (warp 0 reads it only after the first iteration's barrier)
    hess_inverse_block<M, NT>(sm.L, sm.dsc, sm.Hi, tid);

    // ---- ICGN iterations --------------------------------------------------
    const double size = sqrt(dn);
    const double inv_dn = 1.0 / dn, inv_df = 1.0 / df;
    int iters = 0, status = GPV_OK;
    bool converged = false;
    double c_zncc = 0.0, c_znssd = 4.0, last_norm = 0.0, gm_last = 0.0, dg_last = 0.0;
    for (int it = 1; it <= A.max_iter; it++) {
        // (re)stage g's window when the warped square has left it
        const int4 ext = run_extent<ORDER>(sm.p, cx, cy, re, A.w, A.h);
        const bool inside = ext.x & kInside;
        if (!run_covers(sm, ext.x & ~kInside, ext.y, ext.z, ext.w, B)) {
            __syncthreads();  // nobody still reads the old window (or its place)
            place_window<NT>(sm, A.g32, A.pitch32, ch, B, R.win_cap, ext.x & ~kInside, ext.y, ext.z, ext.w, win, 0);
            __syncthreads();
        }
        const bool staged = sm.win_ok != 0;
        const int gr0 = sm.win_r0, gc0 = sm.win_c0, gwh = sm.win_h, gww = sm.win_w, gP = sm.win_p;
        const double X0 = cx + sm.p[0], Y0 = cy + sm.p[1];
        const double bxd = floor(X0), byd = floor(Y0);
        const int wbx = (int)bxd, wby = (int)byd;
        const float ox = (float)(X0 - bxd), oy = (float)(Y0 - byd);
        float ux = 0.f, uy = 0.f, vx = 0.f, vy = 0.f, uxx = 0.f, uxy = 0.f, uyy = 0.f, vxx = 0.f, vxy = 0.f, vyy = 0.f;
        if (ORDER >= 1) { ux = (float)sm.p[2]; vx = (float)sm.p[3]; uy = (float)sm.p[4]; vy = (float)sm.p[5]; }
        if (ORDER == 2) {
            uxx = (float)(0.5 * sm.p[6 % M]); vxx = (float)(0.5 * sm.p[7 % M]); uxy = (float)sm.p[8 % M];
            vxy = (float)sm.p[9 % M]; uyy = (float)(0.5 * sm.p[10 % M]); vyy = (float)(0.5 * sm.p[11 % M]);
        }
        // window-relative origin: integer position (ix, iy) relative to (wbx,
        // wby) reads rows iy + wy0 .., columns ix + wx0 ..
        const int wy0 = wby + B - 2 - gr0, wx0 = wbx + B - 2 - gc0;
        const bool fast = staged && inside;
        // A sample's position relative to (wbx, wby) is its integer offset
        // (dx, dy) plus the small part s(dx, dy) = A2(dx) + B2(dx) dy + C2 dy^2
        // ((y, x) pairs; |s| ~ the fraction plus the deformation over the
        // subset): s is rounded in FP32 at its own small magnitude, and the
        // integer offsets join its floor exactly.
        // (half a pixel lower on the fast path, where floors come by rounding;
        // with the diagnostic the half comes off after: it follows the
        // parameters' last bits, 1e-8 px of another rounding moved it by 5e-6
        // of its size)
        const float half = fast && !ETA ? 0.5f : 0.f;
        const uint32_t o0 = 0u - kMagicBits * ((uint32_t)gP + 1u);
        const float2 O2 = make_float2(oy - half, ox - half), U1 = make_float2(vx, ux), U2 = make_float2(vy, uy);
        const float2 Q1 = make_float2(vxx, uxx), Q2 = make_float2(vxy, uxy), C2 = make_float2(vyy, uyy);
        if constexpr (RIGID) {
            if (rigid_on) {
                // Template pass: G(E(p)) per pixel (grain_template,
                // src/texture.rs:213-244), zero outside the template, and the
                // sums of G, t^2 and SDI_j G (t = f - f_m + G).  The template's
                // mean and gradient are the setup's fixed FP64 sums plus these,
                // which scale with the strain, so their FP32 rounding vanishes
                // with it.  Its spread is its own sum: as a difference of sums of
                // f^2, f G and G^2 a strain that cancels f (its trace 1, where
                // the pixels have no grain) left their rounding, or 0.
                const float s2f = (float)A.grain_scal[2], fmsf = (float)((double)shift - fm);
                const float2 px2 = make_float2(ORDER == 2 ? (float)sm.p[6 % M] : 0.f, ORDER == 2 ? (float)sm.p[7 % M] : 0.f);
                const float2 pxy = make_float2(ORDER == 2 ? (float)sm.p[8 % M] : 0.f, ORDER == 2 ? (float)sm.p[9 % M] : 0.f);
                const float2 py2 = make_float2(ORDER == 2 ? (float)sm.p[10 % M] : 0.f, ORDER == 2 ? (float)sm.p[11 % M] : 0.f);
                double g1 = 0.0, t2 = 0.0;
                KSum unused[3];
                float2 TB[6];
#pragma unroll
                for (int k = 0; k < 6; k++) TB[k] = make_float2(0.f, 0.f);
#pragma unroll 1
                for (int t = tid; t < T; t += NT) {
                    int dx, dy0;
                    unpack_task(tasks[t], dx, dy0);
                    const float dxf = (float)dx;
                    RunAcc ac;
                    ac.p1 = ac.p2 = ac.pfg = 0.f;
                    ac.m0 = ac.m1 = ac.m2 = make_float2(0.f, 0.f);
                    float tt = 0.f;
                    // the run's records and grain samples together in flight (the
                    // stores of G below would order the loads after them)
                    float4 rcs[K];
                    float hs[K][3];
#pragma unroll
                    for (int j = 0; j < K; j++) {
                        rcs[j] = ld_rec(REC + j * T + t);
#pragma unroll
                        for (int m = 0; m < 3; m++) hs[j][m] = ld_once(RH + m * R.nslot + j * T + t);
                    }
#pragma unroll
                    for (int j = 0; j < K; j++) {
                        const int sl = j * T + t;
                        float4 rc = rcs[j];
                        const float h0 = hs[j][0], h1 = hs[j][1], h2 = hs[j][2];
                        const float dyf = (float)(dy0 + j);
                        // (u, v) gradients along x and y at the pixel
                        float gux = ux, gvx = vx, guy = uy, gvy = vy;
                        if (ORDER == 2) {
                            gux = fmaf(px2.x, dxf, fmaf(pxy.x, dyf, ux));
                            gvx = fmaf(px2.y, dxf, fmaf(pxy.y, dyf, vx));
                            guy = fmaf(pxy.x, dxf, fmaf(py2.x, dyf, uy));
                            gvy = fmaf(pxy.y, dxf, fmaf(py2.y, dyf, vy));
                        }
                        float e0, e1, e2;
                        green_lagrange(gux, gvx, guy, gvy, e0, e1, e2);
                        rc.z += fmsf;  // f - f_m
                        const float G = (-0.5f * s2f * (e0 * h0 + e1 * h1 + 2.0f * e2 * h2) - (e0 + e1) * rc.z) * rc.w;
                        RTG[sl] = G;
                        const float tm = fmaf(rc.z, rc.w, G);
                        tt = fmaf(tm, tm, tt);
                        acc_sample<ORDER, false>(ac, unused, rc, G, 0.f, make_float2(dyf, dyf), make_float2(dyf * dyf, dyf * dyf));
                    }
                    g1 += (double)ac.p1;
                    t2 += (double)tt;
                    acc_expand<ORDER>(ac, dxf, TB);
                }
                double *dst = sm.red2[wid];
                const double gv[2] = {g1, t2};
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const double t = warp_sum(gv[q]);
                    if (lane == q) dst[q] = t;
                }
                float tb[M];
#pragma unroll
                for (int j = 0; j < M / 2; j++) {
                    tb[2 * j] = TB[j].x;
                    tb[2 * j + 1] = TB[j].y;
                }
                run_warp_sums<M, false>(tb, sm.part[wid], dst + 3, lane);
            }
        }
        double s1 = 0.0, s2 = 0.0, sfg = 0.0;
        KSum ks[3];
        float2 PB[6];
        float2 PH[6];  // 64 threads: the first of the two sums a thread takes (as at setup)
#pragma unroll
        for (int k = 0; k < 6; k++) PB[k] = PH[k] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int hf = 0; hf < kHalves; hf++) {
        if (hf) {
#pragma unroll
            for (int k = 0; k < M / 2; k++) {
                PH[k] = PB[k];
                PB[k] = make_float2(0.f, 0.f);
            }
        }
        for (int t = hf * NT + tid; t < T; t += kHalves * NT) {
            int dx, dy0;
            unpack_task(tasks[t], dx, dy0);
            const float dxf = (float)dx;
            float2 A2 = O2, B2 = make_float2(0.f, 0.f);
            if (ORDER >= 1) {
                A2 = __ffma2_rn(U1, make_float2(dxf, dxf), A2);
                B2 = U2;
            }
            if (ORDER == 2) {
                A2 = __ffma2_rn(Q1, make_float2(dxf * dxf, dxf * dxf), A2);
                B2 = __ffma2_rn(Q2, make_float2(dxf, dxf), B2);
            }
            RunAcc ac;
            ac.p1 = ac.p2 = ac.pfg = 0.f;
            ac.m0 = ac.m1 = ac.m2 = make_float2(0.f, 0.f);
            if (fast) {
                // no edge clamp can apply and the window covers every tap: the
                // block of coefficients rolls down the run in registers
                float Rg[6][6];
                int py = 0, px = 0;  // floors of the sample before (biased)
                uint32_t off = o0 + (uint32_t)((dy0 + wy0) * gP + dx + wx0);
                const float4 *rec = REC + t;
                float2 dy2 = make_float2((float)dy0, (float)dy0);
#pragma unroll
                for (int j = 0; j < K; j++) {
                    float4 rc = ld_rec(rec);
                    if (RIGID && rigid_on) rc.z += ld_once(RTG + j * T + t);  // the cross term against the template
                    float2 L = A2;
                    const float2 dd2 = __fmul2_rn(dy2, dy2);
                    if (ORDER >= 1) L = __ffma2_rn(B2, dy2, L);
                    if (ORDER == 2) L = __ffma2_rn(C2, dd2, L);
                    // L is half a pixel below the position: rounding to
                    // nearest gives its floor, and u = fraction - 1/2
                    const float2 mh = make_float2(-0.5f, -0.5f);
                    const float2 Mg = __fadd2_rn(ETA ? __fadd2_rn(L, mh) : L, make_float2(kMagic, kMagic));
                    float2 u2 = __fadd2_rn(L, __ffma2_rn(Mg, make_float2(-1.f, -1.f), make_float2(kMagic, kMagic)));
                    if (ETA) u2 = __fadd2_rn(u2, mh);
                    const int iy = __float_as_int(Mg.x), ix = __float_as_int(Mg.y);
                    const float *rp = win + (int)(off + (uint32_t)iy * (uint32_t)gP + (uint32_t)ix);
                    if (j == 0 || ix != px || iy != py) {  // the block did not move down one row: (re)load
#pragma unroll
                        for (int rr = 0; rr < 5; rr++)
#pragma unroll
                            for (int k = 0; k < 6; k++) Rg[(j + rr) % 6][k] = rp[rr * gP + k];
                    }
#pragma unroll
                    for (int k = 0; k < 6; k++) Rg[(j + 5) % 6][k] = rp[5 * gP + k];
                    py = iy;
                    px = ix;
                    float2 Aw[3], Bw[3];
                    basis_sym(u2.y, Bw);
                    float sr[6];
#pragma unroll
                    for (int rr = 0; rr < 6; rr++) sr[rr] = row_dot(Rg[(j + rr) % 6], Bw);
                    basis_sym(u2.x, Aw);
                    const float g = combine6(sr, Aw);
                    acc_sample<ORDER, KAHAN>(ac, ks, rc, g, fmf, dy2, dd2);
                    rec += T;
                    off += (uint32_t)gP;
                    dy2 = __fadd2_rn(dy2, make_float2(1.f, 1.f));
                }
            } else {
#pragma unroll 1
                for (int j = 0; j < K; j++) {
                    const float dyf = (float)(dy0 + j);
                    float2 L = A2;
                    if (ORDER >= 1) L = __ffma2_rn(B2, make_float2(dyf, dyf), L);
                    if (ORDER == 2) L = __ffma2_rn(C2, make_float2(dyf * dyf, dyf * dyf), L);
                    int ix, iy;
                    float tx, ty;
                    split_clamped(wbx + dx, L.y, A.w, ix, tx);
                    split_clamped(wby + dy0 + j, L.x, A.h, iy, ty);
                    float a[6], b[6];
                    basis(ty, a);
                    basis(tx, b);
                    float g;
                    if (staged) {
                        const int wx = min(max(ix + B - 2 - gc0, 0), gww - 6), wy = min(max(iy + B - 2 - gr0, 0), gwh - 6);
                        g = contract<float>(win + wy * gP + wx, gP, a, b);
                    } else {
                        g = contract<float>(A.g32 + (int64_t)(iy + B - 2) * A.pitch32 + (ix + B - 2), A.pitch32, a, b);
                    }
                    const int sl = j * T + t;
                    float4 rc = REC[sl];
                    if (RIGID && rigid_on) rc.z += RTG[sl];
                    acc_sample<ORDER, KAHAN>(ac, ks, rc, g, fmf, make_float2(dyf, dyf), make_float2(dyf * dyf, dyf * dyf));
                }
            }
            if (!KAHAN) {
                s1 += (double)ac.p1;
                s2 += (double)ac.p2;
                sfg += (double)ac.pfg;
            }
            acc_expand<ORDER>(ac, dxf, PB);
        }
        }
        // block sums: warp partials to shared memory, one barrier, then warp 0
        // adds them up and updates the warp; a second barrier publishes p
        constexpr int KR = 3 + M;
        {
            double v[3] = {s1, s2, sfg};
            if (KAHAN) {
                v[0] = ks[0].s;
                v[1] = ks[1].s;
                v[2] = ks[2].s;
            }
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const double t = warp_sum(v[q]);
                if (lane == q) sm.red[wid][q] = t;
            }
            float pb[kHalves * M];  // both sums of 64 threads, joined in FP64 below
#pragma unroll
            for (int j = 0; j < M / 2; j++) {
                pb[2 * j] = PB[j].x;
                pb[2 * j + 1] = PB[j].y;
                if constexpr (kHalves == 2) {
                    pb[M + 2 * j] = PH[j].x;
                    pb[M + 2 * j + 1] = PH[j].y;
                }
            }
            run_warp_sums<kHalves * M, false>(pb, sm.part[wid], kHalves == 2 ? sm.red2[wid] : sm.red[wid] + 3, lane);
        }
        __syncthreads();
        if (wid == 0) {
            double tl = 0.0;
            if (lane < KR) {
                if (kHalves == 2 && lane >= 3) {
#pragma unroll
                    for (int w = 0; w < NT / 32; w++) tl += sm.red2[w][lane - 3] + sm.red2[w][lane - 3 + M];
                } else {
#pragma unroll
                    for (int w = 0; w < NT / 32; w++) tl += sm.red[w][lane];
                }
            }
            const double t0 = __shfl_sync(0xffffffffu, tl, 0), t1 = __shfl_sync(0xffffffffu, tl, 1);
            const double t2 = __shfl_sync(0xffffffffu, tl, 2);
            const double gmt = t0 * inv_dn;
            const double dg2 = t1 - t0 * gmt;
            const double dg2p = dg2 > 0.0 ? dg2 : 0.0;
            // sum (f - f_m)(g - g_m) = sum (f - f_m)(g - f_m) (sum (f - f_m) = 0)
            //                     = sum (f - s)(g - f_m) - (f_m - s) sum (g - f_m)
            double sab = t2 - (fm - (double)shift) * t0;
            double dref = df, inv_dref = inv_df, tmf = 0.0, sgj = 0.0;
            if constexpr (RIGID) {
                if (rigid_on) {  // against the template t = f + G: t_m = f_m + tmf, spread dref
                    double tq = 0.0;
                    if (lane < KR) {
#pragma unroll
                        for (int w = 0; w < NT / 32; w++) tq += sm.red2[w][lane];
                    }
                    const double q0 = __shfl_sync(0xffffffffu, tq, 0), q1 = __shfl_sync(0xffffffffu, tq, 1);
                    sgj = __shfl_down_sync(0xffffffffu, tq, 3);  // lane j: sum SDI_j G
                    tmf = q0 * inv_dn;
                    const double dt2 = q1 - q0 * tmf;
                    dref = sqrt(dt2 < 0.0 ? 0.0 : dt2);
                    inv_dref = dref > 0.0 ? 1.0 / dref : __longlong_as_double(0x7ff8000000000000ll);  // no template, no ZNCC
                    sab -= tmf * t0;
                }
            }
            const double rdg = rsqrt(dg2p);  // 1 / delta_g: one reciprocal square root on the update's critical path
            const double dg = dg2p > 0.0 ? dg2p * rdg : 0.0;
            const double znssd = 2.0 - 2.0 * sab * (inv_dref * rdg);
            const double ratio = dref * rdg;
            // lane j < M: grad_j = A_j - (df/dg)(B_j - g~_m S_j); B_j sits at lane 3 + j
            const double bj = __shfl_down_sync(0xffffffffu, tl, 3);
            const double gj = lane < M ? sm.A[lane] + (RIGID ? sgj - tmf * sm.S[lane] : 0.0) - ratio * (bj - gmt * sm.S[lane]) : 0.0;
            // dp = -H^-1 grad with the inverse formed from the Cholesky factor at setup
            // (12 lanes, two FMA chains each; 1.7% faster than two substitutions)
            if (lane < M) sm.grad[lane] = gj;
            __syncwarp();
            double dpj = 0.0;
            if (lane < M) {
                double a0 = 0.0, a1 = 0.0;
#pragma unroll
                for (int k = 0; k < M; k += 2) {
                    a0 = fma(sm.Hi[lane * M + k], sm.grad[k], a0);
                    if (k + 1 < M) a1 = fma(sm.Hi[lane * M + k + 1], sm.grad[k + 1], a1);
                }
                dpj = -(a0 + a1);
            }
            if (lane < M) {
                sm.dp[lane] = dpj;
                sm.pprev[lane] = sm.p[lane];
            }
            // convergence_norm (src/subset.rs:622-649), a term per lane
            double nt = lane < M ? dpj * (lane < 2 ? 1.0 : (lane < 6 ? size : 0.5 * dn)) : 0.0;
            nt *= nt;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) nt += __shfl_down_sync(0xffffffffu, nt, o);
            __syncwarp();
            if (lane == 0) {
                double pn[12], dpl[12], pl[12];
#pragma unroll
                for (int k = 0; k < 12; k++) {
                    dpl[k] = sm.dp[k % M];
                    pl[k] = sm.p[k % M];
                }
                bool ok = true;
                if (ORDER == 0) {
                    pn[0] = pl[0] - dpl[0];
                    pn[1] = pl[1] - dpl[1];
                } else if (ORDER == 1) {
                    ok = compose1(pl, dpl, pn);
                } else {
                    ok = compose2_regs(pl, dpl, pn);
                }
                if (ok) {
#pragma unroll
                    for (int k = 0; k < M; k++) sm.p[k] = pn[k];
                }
                sm.flag[1] = ok;
                sm.misc[1] = sqrt(nt);
                sm.misc[2] = gmt;
                sm.misc[3] = dg;
                sm.misc[4] = znssd;
            }
        }
        __syncthreads();
        const double gmt = sm.misc[2], dg = sm.misc[3], znssd = sm.misc[4];
        gm_last = fm + gmt;
        dg_last = dg;
        if (!sm.flag[1]) {
            status = GPV_SINGULAR_WDELTA;  // p keeps the last valid warp
            break;
        }
        const double nrm = sm.misc[1];
        c_znssd = znssd;
        c_zncc = 1.0 - znssd / 2.0;
        iters = it;
        last_norm = nrm;
        if (tid == 0) write_history(A, idx, it, nrm, c_zncc, c_znssd);
        if (!isfinite(nrm)) { status = GPV_NONFINITE; break; }
        if (nrm < A.max_norm) { converged = true; break; }
    }

    // ---- eta diagnostic at the last sampled warp (optional) -----------------
    double eu = 0.0, ev = 0.0;
    const bool want_eta = ETA && iters > 0 && status == GPV_OK;
    if constexpr (ETA) {
        if (want_eta)
            run_eta<ORDER, NT, K>(sm, win, A.g32, A.pitch32, A.w, A.h, B, tasks, T, REC, RSG, RVM, cx, cy, (double)shift - fm,
                              dn, df, gm_last, dg_last, &eu, &ev);
    }
    if (tid == 0) {
        gpv_subset_result *o = A.out + idx;
#pragma unroll
        for (int k = 0; k < 12; k++) o->p[k] = k < M ? sm.p[k % M] : 0.0;
        o->c_zncc = c_zncc;
        o->c_znssd = c_znssd;
        o->norm = last_norm;
        o->eta_u = eu;
        o->eta_v = ev;
        o->f_m = fm;
        o->delta_f = df;
        o->sssig = tot_sssig;
        o->sigma = sqrt(saa / dn);
        o->iterations = iters;
        o->converged = converged;
        o->quality_ok = converged && c_zncc >= A.tolerance;
        o->status = status;
        o->n_px = n;
        o->has_eta = want_eta;
        o->texture = rigid_on ? 1 : 0;
        o->reserved = 0;
    }
}

// Claim a free scratch slot of the SM this block runs on (one block per
// subset): at most slots_per_sm blocks of a launch are resident on an SM
// and each frees its slot before it exits, so a bit is free when a block
// starts; the bounded wait only covers a block moved to another SM after a
// preemption.  -1: none claimed.
__device__ int run_claim_slot(const RunArgs &R) {
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    if ((int)smid >= R.n_mask) return -1;
    for (int attempt = 0; attempt < 20000; attempt++) {
        for (int j = 0; j < R.slots_per_sm; j++) {
            const unsigned bit = 1u << j;
            if (!(atomicOr(R.slot_mask + smid, bit) & bit)) return (int)smid * R.slots_per_sm + j;
        }
        __nanosleep(1000);
    }
    return -1;
}

// PER_SUBSET: one block per subset with a claimed scratch slot (subsets
// free SMs one at a time, for callers sharing the GPU); else a persistent
// grid whose blocks take subsets of their segment from the queue.
template <int ORDER, int NT, int K, bool PER_SUBSET, bool KAHAN, bool ETA, bool RIGID>
__global__ void __launch_bounds__(NT, 512 / NT) icgn_runs(RunArgs R) {
    extern __shared__ float4 win4[];
    float *win = reinterpret_cast<float *>(win4);
    __shared__ RunSmem<NT / 32> sm;
    const KArgs &A = R.k;
    const int start = R.seg[0], count = R.seg[1];
    if (PER_SUBSET) {
        const int item = blockIdx.x;
        if (item >= count) return;
        if (threadIdx.x == 0) sm.item = run_claim_slot(R);
        __threadfence();
        __syncthreads();
        const int slot = sm.item;
        const int idx = A.order[start + item];
        const gpv_subset_desc d = A.desc[idx];
        if (slot < 0) {
            if (threadIdx.x == 0) write_failed(A, idx, d, 12, GPV_TIMEOUT, 0, 0.0, 0.0);
            return;
        }
        float *base = reinterpret_cast<float *>(A.scratch) + (int64_t)slot * A.scratch_stride;
        if (d.radius < 1 || d.radius > A.max_radius) {
            if (threadIdx.x == 0) write_failed(A, idx, d, 12, GPV_INVALID_SUBSET, 0, 0.0, 0.0);
        } else {
            run_subset<ORDER, NT, K, KAHAN, ETA, RIGID>(R, idx, d, base, win, sm);
        }
        __threadfence();  // every scratch access of the block is done before the slot is free
        __syncthreads();
        if (threadIdx.x == 0) {
            const int own = sm.item;
            atomicAnd(R.slot_mask + own / R.slots_per_sm, ~(1u << (own % R.slots_per_sm)));
        }
        return;
    }
    float *base = reinterpret_cast<float *>(A.scratch) + (int64_t)blockIdx.x * A.scratch_stride;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) sm.item = atomicAdd(R.queue, 1);
        __syncthreads();
        const int item = sm.item;
        if (item >= count) break;
        const int idx = A.order[start + item];
        const gpv_subset_desc d = A.desc[idx];
        if (d.radius < 1 || d.radius > A.max_radius) {
            if (threadIdx.x == 0) write_failed(A, idx, d, 12, GPV_INVALID_SUBSET, 0, 0.0, 0.0);
            continue;
        }
        run_subset<ORDER, NT, K, KAHAN, ETA, RIGID>(R, idx, d, base, win, sm);
    }
}

// Instantiations: every (threads, one block per subset, with or without the
// diagnostic); the compensated-sum form and the rigid-texture template (orders
// 1 and 2, without the diagnostic) on persistent grids of 128 or 256 threads only.
template <int NT, bool PS, bool KH, bool ETA>
const void *run_kernel_t(int order) {
    return order == 2 ? (const void *)icgn_runs<2, NT, kRunK, PS, KH, ETA, false>
                      : (order == 1 ? (const void *)icgn_runs<1, NT, kRunK, PS, KH, ETA, false>
                                    : (const void *)icgn_runs<0, NT, kRunK, PS, KH, ETA, false>);
}

template <int NT>
const void *run_kernel_rigid(int order) {
    return order == 2 ? (const void *)icgn_runs<2, NT, kRunK, false, false, false, true>
                      : (const void *)icgn_runs<1, NT, kRunK, false, false, false, true>;
}

template <int NT>
const void *run_kernel_nt(int order, RunForm form, bool eta) {
    if constexpr (NT >= 128) {
        if (form == RunForm::kRigid) return run_kernel_rigid<NT>(order);
        if (form == RunForm::kKahan) return eta ? run_kernel_t<NT, false, true, true>(order) : run_kernel_t<NT, false, true, false>(order);
    }
    if (form == RunForm::kPerSubset) return eta ? run_kernel_t<NT, true, false, true>(order) : run_kernel_t<NT, true, false, false>(order);
    return eta ? run_kernel_t<NT, false, false, true>(order) : run_kernel_t<NT, false, false, false>(order);
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side: run tables, sizes and launches (called by the batched launcher).
// ---------------------------------------------------------------------------

// Window capacity (floats) of a launch for subsets up to radius rmax: the
// square of half side max(rmax, kRunK - 1 - rmax) stretched by 6%, taps and
// margins, at a pitch of whole 32-float rows.
int run_window_cap(int rmax) {
    const int e = std::max(rmax, kRunK - 1 - rmax);
    const int rw = (int)std::ceil(1.06 * e) + 2;
    const int side = 2 * rw + 6 + 2 * kRunMargin + 4;
    return side * run_pitch<32>(side);
}

// Record slots per block (largest radius's runs x kRunK, rounded to 32) and the
// scratch floats per block: a float4 record and an eta resample per slot, one
// word of pixel bits per run; for the rigid template three grain samples and
// the correction per slot.
int64_t run_scratch_floats(gpv_context *ctx, int rmax, bool rigid, int *nslot) {
    int T = 0;  // the most runs of any radius up to rmax (the count is not monotone in r)
    for (int r = 1; r <= rmax; r++) T = std::max(T, (int)ctx->h_run_n[r]);
    const int ns = (T * kRunK + 31) / 32 * 32;
    *nslot = ns;
    return run_plain_floats(ns) + (rigid ? 4 * (int64_t)ns : 0);
}

const void *run_kernel(int order, int nt, RunForm form, bool eta) {
    if (nt == 64) return run_kernel_nt<64>(order, form, eta);
    return nt == 256 ? run_kernel_nt<256>(order, form, eta) : run_kernel_nt<128>(order, form, eta);
}

int run_launch(gpv_context *ctx, const void *fn, int nt, int blocks, size_t smem, cudaStream_t s, const KArgs &k,
               const int32_t *seg, int *queue, int win_cap, int nslot, uint32_t *slot_mask, int slots_per_sm, int n_mask) {
    RunArgs R;
    R.k = k;
    run_tables(ctx, R);
    R.seg = seg;
    R.queue = queue;
    R.win_cap = win_cap;
    R.nslot = nslot;
    R.slot_mask = slot_mask;
    R.slots_per_sm = slots_per_sm;
    R.n_mask = n_mask;
    void *args[] = {&R};
    GPV_CUDA_TRY(cudaLaunchKernel(fn, dim3((unsigned)blocks), dim3((unsigned)nt), args, smem, s));
    return GPV_SUCCESS;
}

}  // namespace gpv
