// icgn_runs64.cu -- the FP64 subset solves with the circular template cut
// into vertical runs: inverse-compositional Gauss-Newton on FP64
// coefficients, and forward additive Gauss-Newton (FP64 arithmetic on FP64 or
// FP32 coefficients).
//
// Subset::new (src/subset.rs:836-919), solve_icgn_result (:1117-1219) and
// solve_fagn_result (:1228-1334), with the layout of the mixed-precision run
// kernel (icgn_runs.cu): one block per subset at a time on a persistent grid,
// the windows of the coefficients staged in shared memory as doubles, a lane
// walking runs of K vertically adjacent template pixels with the 6 x 6 block
// of the current sample rolled through registers.  What bounds it is the FP64
// pipe (about 64 multiply-adds a clock and SM): a target sample takes 42
// multiply-adds of taps, 40 of basis weights and about 25 of positions and
// sums.  Reading every tap from shared memory would take 72 clocks of its
// bandwidth per 32 samples against about 55 of the FP64 pipe; the rolled block
// takes 12.
//
//  * ICGN takes one sweep per iteration: about a level c (the target's mean of
//    the iteration before, f's mean at first) it sums b = g - c, b^2, a b
//    (a = f - f_m), e^2 (e = a - rho b, rho = delta_f / delta_g of the
//    iteration before) and SDI_j e.  With t = delta_f / delta_g,
//    k = t - rho and d the mean of b,
//        residual r = a - t (b - d) = e - k b + t d
//        grad_j   = sum SDI_j e - k sum SDI_j b + t d sum SDI_j,
//                   sum SDI_j b = (sum SDI_j a - sum SDI_j e) / rho
//        ZNSSD    = sum r^2 / delta_f^2,
//    where sum r^2 follows from sum e^2 and small corrections (k and d go to
//    zero as the solve converges), so ZNSSD and the gradient keep the relative
//    accuracy of the direct sums over the residual (a difference of sums of
//    SDI_j a and SDI_j b cost an ill-conditioned subset 1e-5 px).  That costs digits where the target's level is far from c against
//    its contrast (a first iteration on a target of another brightness, or
//    one without contrast), rho far above t, or a Hessian near singular (few
//    pixels: only the direct sum's rounding stays where its inverse is small):
//    there three more sweeps take the mean, the spread about it and the direct sums.
//  * FAGN takes two sweeps: target value and gradient at the warped positions
//    (kept per pixel), then the Hessian's moments and the residual gradient
//    about the warped centre.
//  * The Hessian is factored by one warp (hess_factor); a matrix with a scaled
//    pivot of kMinPivot or less (rank-deficient to rounding, where a residue would pass
//    for a pivot, or nearly so) goes to the pivoted elimination (gj_inverse),
//    so only what that rejects is singular.  Second-order composition eliminates without
//    pivoting while the pivots stay near 1, else with pivoting.
// Measured against one sweep-per-sum block of 256 threads with taps through L1
// (icgn_fp64, fagn_kernel; 254 registers, 8 warps per SM, FP64 pipe 14 % and
// 29 % busy): 8,836 second-order subsets of radius 30 12.53 -> 2.28 ms (FP64
// pipe 46 %), 2,304 first-order FAGN solves of radius 25 on FP32 coefficients
// 1.27 -> 0.63 ms (48 %).
// Samples that can meet the image's edge, and windows that do not fit in
// shared memory, take a clamped per-sample path (src/image.rs:129-132).
#include <algorithm>
#include <cmath>

#include "icgn_runs.cuh"

namespace gpv {
namespace {

constexpr int kK = kRunK;
// The sums about a level are used while they leave the spread all but two of
// its digits (a target ten times its contrast away from the level), and the
// residual's sum while the scale of the iteration before is within 32 times the new one.
constexpr double kMinPivot = 1e-10;  // about the square root of a rounding's share of the unit diagonal, and less
constexpr double kLevelDigits = 0.01, kScaleDigits = 32.0 * 32.0;

template <int NW>
struct Smem64 {
    double mom[3 * 15];
    double L[144];   // the factor's inverse
    double Hi[160];  // the factor, then H^-1
    double linv[12], dsc[12];
    double A[12], S[12];
    double p[12], pprev[12], dp[12], grad[12];
    double red[NW][16];
    double red2[NW][80];
    double tot[80];
    double misc[12];
    int flag[4];
    int item;
    int n_valid;
    int win_r0, win_c0, win_h, win_w, win_p, win_ok;
};

// Coefficient rows [r0, r0 + wh) x columns [c0, c0 + ww) (c0, ww multiples of
// 4) into win as doubles, out-of-range rows / columns clamped, by threads
// [t0, NT).  FP64 coefficients by 16-byte cp.async (rows are a multiple of 16
// doubles apart, c0, the clamped columns and the pitch even); FP32 ones are
// read as float4 and widened once here instead of at every tap.
template <int NT, typename C>
__device__ __forceinline__ void stage64(const C *__restrict__ coef, int64_t cpitch, int ch, int r0, int c0, int wh, int ww,
                                        int pitch, double *win, int t0) {
    constexpr int V = sizeof(C) == 8 ? 2 : 4;
    const int nv = ww / V;
    for (int idx = (int)threadIdx.x - t0; idx < wh * nv; idx += NT - t0) {
        const int rr = idx / nv, cc = (idx - rr * nv) * V;
        const int row = min(max(r0 + rr, 0), ch - 1);
        const int col = min(max(c0 + cc, 0), (int)cpitch - V);
        const C *src = coef + (int64_t)row * cpitch + col;
        double *dst = win + rr * pitch + cc;
        if (V == 2) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                         : "memory");
        } else {
            const float4 v = *reinterpret_cast<const float4 *>(src);
            *reinterpret_cast<double2 *>(dst) = make_double2(v.x, v.y);
            *reinterpret_cast<double2 *>(dst + 2) = make_double2(v.z, v.w);
        }
    }
    if (V == 2) asm volatile("cp.async.wait_all;\n" ::: "memory");
}

template <int NT>
__device__ double block_sum64(double v, Smem64<NT / 32> &sm) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const double s = warp_sum(v);
    __syncthreads();
    if (lane == 0) sm.red[wid][0] = s;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < NT / 32; w++) t += sm.red[w][0];
    return t;
}

// The weights of basis() with the odd part joined by a fused multiply-add.
__device__ __forceinline__ void weights64(double t, double (&w)[6]) {
    const double u = t - 0.5, v = u * u;
    const double e0 = fma(fma(v, 1.0 / 48.0, 1.0 / 96.0), v, 1.0 / 3840.0);
    const double e1 = fma(fma(v, -1.0 / 16.0, 7.0 / 32.0), v, 79.0 / 1280.0);
    const double e2 = fma(fma(v, 1.0 / 24.0, -11.0 / 48.0), v, 841.0 / 1920.0);
    const double q0 = fma(fma(v, 1.0 / 120.0, 1.0 / 48.0), v, 1.0 / 384.0);
    const double q1 = fma(fma(v, -1.0 / 24.0, 1.0 / 16.0), v, 25.0 / 128.0);
    const double q2 = fma(fma(v, 1.0 / 12.0, -7.0 / 24.0), v, 77.0 / 192.0);
    w[0] = fma(-u, q0, e0); w[5] = fma(u, q0, e0);
    w[1] = fma(-u, q1, e1); w[4] = fma(u, q1, e1);
    w[2] = fma(-u, q2, e2); w[3] = fma(u, q2, e2);
}

__device__ __forceinline__ double dot6(const double (&c)[6], const double (&b)[6]) {
    // two chains of three: half the latency of one chain of six
    return fma(c[4], b[4], fma(c[2], b[2], c[0] * b[0])) + fma(c[5], b[5], fma(c[3], b[3], c[1] * b[1]));
}

// One chain, in the taps' order: on equal coefficients the two chains of dot6
// cancel a derivative's weights to exactly 0 (a saturated target would have a
// singular FAGN Hessian), this one to its rounding as contract_grad does.
__device__ __forceinline__ double seq6(const double (&c)[6], const double (&b)[6]) {
    return fma(c[5], b[5], fma(c[4], b[4], fma(c[3], b[3], fma(c[2], b[2], fma(c[1], b[1], c[0] * b[0])))));
}

// split_clamped for the warped positions, which may lie past the range of an int:
// base (whole) and floor(loc) are added in FP64.
__device__ __forceinline__ void split_far(double base, double loc, int n, int &i, double &t) {
    const double fl = floor(loc), at = base + fl;
    t = loc - fl;
    i = (int)at;  // a NaN gives 0, and t is NaN
    if (at < 0.0) {
        i = 0;
        t = 0.0;
    } else if (at > (double)(n - 1)) {
        i = n - 1;
        t = 1.0 - 1e-9;
    }
}

// A record's parts, read once per sweep: not kept in L1.
__device__ __forceinline__ double2 ld_pair(const double2 *p) {
    double2 v;
    asm volatile("ld.global.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_one(const double *p) {
    double v;
    asm volatile("ld.global.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Gauss-Jordan inverse with partial pivoting by one thread, for matrices that
// the Cholesky factor rejects; false when no pivot is left.
template <int M>
__device__ __noinline__ bool gj_inverse(double *a, double *inv) {
    for (int e = 0; e < M * M; e++) inv[e] = (e / M == e % M) ? 1.0 : 0.0;
    for (int k = 0; k < M; k++) {
        int piv = k;
        double best = fabs(a[k * M + k]);
        for (int i = k + 1; i < M; i++)
            if (fabs(a[i * M + k]) > best) { best = fabs(a[i * M + k]); piv = i; }
        if (!(best > 0.0) || !isfinite(best)) return false;
        if (piv != k)
            for (int j = 0; j < M; j++) {
                double t = a[k * M + j]; a[k * M + j] = a[piv * M + j]; a[piv * M + j] = t;
                t = inv[k * M + j]; inv[k * M + j] = inv[piv * M + j]; inv[piv * M + j] = t;
            }
        const double d = 1.0 / a[k * M + k];
        for (int j = 0; j < M; j++) { a[k * M + j] *= d; inv[k * M + j] *= d; }
        for (int i = 0; i < M; i++) {
            if (i == k) continue;
            const double f = a[i * M + k];
            if (f == 0.0) continue;
            for (int j = 0; j < M; j++) { a[i * M + j] -= f * a[k * M + j]; inv[i * M + j] -= f * inv[k * M + j]; }
        }
    }
    return true;
}

// Second-order composition: without pivoting while every pivot stays within a
// factor of two of 1 (the lifted increment is near unit triangular), else
// the pivoted elimination; ws: 96 doubles.
__device__ __noinline__ bool compose2_any(const double *p, const double *d, double *out, double *ws) {
    double s = 0.0;
    for (int k = 2; k < 12; k++) s = fmax(s, fabs(d[k]));
    s = fmax(s, fmax(fabs(d[0]), fabs(d[1])) * fmax(s, 1e-3));
    if (s < 0.05) return compose2_regs(p, d, out);
    return compose2(p, d, out, ws);
}

// The setup's sums about f's mean, by one warp, from the records: for a level
// (the coefficient under the centre) that is far from the subset's values against
// their contrast, as at a hot pixel that the mask leaves out.  tot[1], tot[2] and
// tot[4 + j] become sum (f - m), sum (f - m)^2 and sum SDI_j (f - m).
template <int ORDER, bool FAGN>
__device__ __noinline__ void sums_about_mean(const double2 *RG, const double *RF, const int *RVM, const int2 *tasks, int T,
                                             double m, double *tot, int lane) {
    constexpr int M = Ord<ORDER>::M, N = FAGN ? 2 : 2 + M;
    double s[N];
#pragma unroll
    for (int q = 0; q < N; q++) s[q] = 0.0;
#pragma unroll 1
    for (int t = lane; t < T; t += 32) {
        int dx, dy0;
        unpack_task(tasks[t], dx, dy0);
        const int vm = RVM[t];
#pragma unroll 1
        for (int j = 0; j < kK; j++) {
            if (!((vm >> j) & 1)) continue;
            const double f = RF[j * T + t], a = f - m;
            if (f != f) continue;  // a subset of NaN alone has f_m NaN and delta_f 0
            s[0] += a;
            s[1] = fma(a, a, s[1]);
            if constexpr (!FAGN) {
                const double2 g = RG[j * T + t];
#pragma unroll
                for (int mu = 0; mu < M / 2; mu++) {
                    const double w = mu_val<double>(mu, dx, dy0 + j) * a;
                    s[2 + 2 * mu] = fma(g.x, w, s[2 + 2 * mu]);
                    s[3 + 2 * mu] = fma(g.y, w, s[3 + 2 * mu]);
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < N; q++) {
        const double v = warp_sum(s[q]);
        if (lane == 0) tot[q < 2 ? 1 + q : 2 + q] = v;
    }
    __syncwarp();
}

// The gradient moments again, by one warp, each pixel's gradient product times
// the whole monomial: where offsets depend on one another (a mask of one line)
// the Hessian's rows then do so to the last bit, as the elimination's test for an
// exact zero needs; the setup's powers of dy per run round in between.
template <int ORDER>
__device__ __noinline__ void moments_of_monomials(const double2 *RG, const int *RVM, const int2 *tasks, int T, double *mom,
                                                  int lane) {
    constexpr int NMOM = Ord<ORDER>::NMOM, NB = 2 * Ord<ORDER>::DEG + 1;
#pragma unroll 1
    for (int pr = 0; pr < 3; pr++) {
        double s[NMOM];
#pragma unroll
        for (int q = 0; q < NMOM; q++) s[q] = 0.0;
#pragma unroll 1
        for (int t = lane; t < T; t += 32) {
            int dx, dy0;
            unpack_task(tasks[t], dx, dy0);
            const int vm = RVM[t];
#pragma unroll 1
            for (int j = 0; j < kK; j++) {
                if (!((vm >> j) & 1)) continue;
                const double2 g = RG[j * T + t];
                const double gg = (pr == 2 ? g.y : g.x) * (pr == 0 ? g.x : g.y);
                double xp = 1.0;
#pragma unroll
                for (int a = 0; a < NB; a++) {
                    double mono = xp;
#pragma unroll
                    for (int b = 0; a + b < NB; b++) {
                        s[mom_idx(a, b)] = fma(gg, mono, s[mom_idx(a, b)]);
                        mono *= dy0 + j;
                    }
                    xp *= dx;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < NMOM; q++) {
            const double v = warp_sum(s[q]);
            if (lane == 0) mom[pr * NMOM + q] = v;
        }
    }
    __syncwarp();
}

// One solve.  scratch (doubles, nslot slots per array, slot j * T + t for
// pixel j of run t): the gradient pair, f, g; for
// FAGN the target's gradient pair too; then one word of pixel bits per run.
template <int ORDER, int NT, bool FAGN, typename C, bool ETA>
__device__ void run64_subset(const RunArgs &R, int idx, const gpv_subset_desc &d, double *base, double *win,
                             Smem64<NT / 32> &sm) {
    const KArgs &A = R.k;
    using O = Ord<ORDER>;
    constexpr int M = O::M, NMU = O::NMU, NMOM = O::NMOM, NB = 2 * O::DEG + 1, NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const C *FC, *GC;
    int64_t cp;
    if constexpr (sizeof(C) == 8) {
        FC = A.f64; GC = A.g64; cp = A.pitch64;
    } else {
        FC = A.f32; GC = A.g32; cp = A.pitch32;
    }
    const int r = d.radius;
    const int re = max(r, kK - 1 - r);
    const int T = R.task_n[r];
    const int2 *tasks = R.tasks + R.task_off[r];
    double2 *RG = reinterpret_cast<double2 *>(base);
    double *RF = base + 2 * (int64_t)R.nslot, *RT = base + 3 * (int64_t)R.nslot;
    double2 *RH = reinterpret_cast<double2 *>(base + 4 * (int64_t)R.nslot);  // FAGN only
    int *RVM = reinterpret_cast<int *>(base + (FAGN ? 6 : 4) * (int64_t)R.nslot);
    const double cx = d.coord[0], cy = d.coord[1];
    const int cxi = (int)cx, cyi = (int)cy;
    const double fxd = floor(cx), fyd = floor(cy);
    const int bx = (int)fxd, by = (int)fyd;
    const double fx = cx - fxd, fy = cy - fyd;
    const int B = A.border, ch = A.h + 2 * B;

    // ---- f's window --------------------------------------------------------
    {
        // +-1: centre fraction plus offset can round up to the next integer
        const int xlo = max(0, min(bx - re - 1, A.w - 1)), xhi = max(0, min(bx + re + 1, A.w - 1));
        const int ylo = max(0, min(by - re - 1, A.h - 1)), yhi = max(0, min(by + re + 1, A.h - 1));
        int r0, c0, wh, ww, pitch;
        const bool ok = run_plan<16>(xlo, xhi, ylo, yhi, B, R.win_cap, r0, c0, wh, ww, pitch);
        if (ok) stage64<NT>(FC, cp, ch, r0, c0, wh, ww, pitch, win, 0);
        if (tid == 0) {
            sm.win_ok = 0;
            sm.win_r0 = r0; sm.win_c0 = c0; sm.win_h = wh; sm.win_w = ww; sm.win_p = pitch;
            sm.flag[2] = ok;
        }
        if (tid < M) {
            sm.p[tid] = d.p0[tid];
            sm.pprev[tid] = d.p0[tid];
        }
        __syncthreads();
    }
    const bool f_staged = sm.flag[2] != 0;
    const int fr0 = sm.win_r0, fc0 = sm.win_c0, fwh = sm.win_h, fww = sm.win_w, fP = sm.win_p;
    const bool interior = f_staged && bx - re >= 0 && bx + re <= A.w - 1 && by - re >= 0 && by + re <= A.h - 1;

    // ---- setup, pass 1: f and its gradient per pixel, first sums ----------
    // [count, sum (f - s), sum (f - s)^2, SSSIG, sum SDI_j (f - s), sum SDI_j]
    constexpr int NVA = FAGN ? 4 : 4 + 2 * M;
    double acc[NVA];
#pragma unroll
    for (int q = 0; q < NVA; q++) acc[q] = 0.0;
    const double shift = (double)FC[(int64_t)(max(0, min(by, A.h - 1)) + B) * cp + max(0, min(bx, A.w - 1)) + B];
    auto pix1 = [&](int sl, bool v, double f, double gx, double gy, double dx, double dy) {
        const double fs = v ? f - shift : 0.0;
        if (!v) gx = gy = 0.0;
        RG[sl] = make_double2(gx, gy);
        RF[sl] = v ? f : 0.0;  // as it is: f - s would lose digits at a far s
        if (!v) return;
        acc[0] += 1.0;
        acc[1] += fs;
        acc[2] = fma(fs, fs, acc[2]);
        acc[3] = fma(0.5 * gx, gx, fma(0.5 * gy, gy, acc[3]));
        if constexpr (!FAGN) {
            const double gxf = gx * fs, gyf = gy * fs;
#pragma unroll
            for (int mu = 0; mu < NMU; mu++) {
                const double mv = mu_val<double>(mu, dx, dy);
                acc[4 + 2 * mu] = fma(gxf, mv, acc[4 + 2 * mu]);
                acc[5 + 2 * mu] = fma(gyf, mv, acc[5 + 2 * mu]);
                acc[4 + M + 2 * mu] = fma(gx, mv, acc[4 + M + 2 * mu]);
                acc[5 + M + 2 * mu] = fma(gy, mv, acc[5 + M + 2 * mu]);
            }
        }
    };
    {
        double a0[6], da0[6], b0[6], db0[6];
        basis(fy, a0); dbasis(fy, da0);
        basis(fx, b0); dbasis(fx, db0);
        for (int t = tid; t < T; t += NT) {
            int dx, dy0;
            unpack_task(tasks[t], dx, dy0);
            uint32_t vm = (uint32_t)tasks[t].y;
            if (A.mask) {
#pragma unroll
                for (int j = 0; j < kK; j++)
                    if (!mask_ok(A, cxi, cyi, dx, dy0 + j)) vm &= ~(1u << j);
            }
            RVM[t] = (int)vm;
            if (interior) {
                // all pixels share one fraction: the run's kK + 5 row sums once, six per pixel
                const double *p0 = win + (by + dy0 + B - 2 - fr0) * fP + (bx + dx + B - 2 - fc0);
                double s[kK + 5], q[kK + 5];
#pragma unroll
                for (int m = 0; m < kK + 5; m++) {
                    const double *rp = p0 + m * fP;
                    double sv = rp[0] * b0[0], qv = rp[0] * db0[0];
#pragma unroll
                    for (int k = 1; k < 6; k++) {
                        sv = fma(rp[k], b0[k], sv);
                        qv = fma(rp[k], db0[k], qv);
                    }
                    s[m] = sv;
                    q[m] = qv;
                }
#pragma unroll
                for (int j = 0; j < kK; j++) {
                    double val = 0.0, vx = 0.0, vy = 0.0;
#pragma unroll
                    for (int rr = 0; rr < 6; rr++) {
                        val = fma(a0[rr], s[j + rr], val);
                        vx = fma(a0[rr], q[j + rr], vx);
                        vy = fma(da0[rr], s[j + rr], vy);
                    }
                    pix1(j * T + t, (vm >> j) & 1u, val, vx, vy, dx, dy0 + j);
                }
            } else {
#pragma unroll 1
                for (int j = 0; j < kK; j++) {
                    int ix, iy;
                    double tx, ty;
                    split_clamped(bx, fx + (double)dx, A.w, ix, tx);
                    split_clamped(by, fy + (double)(dy0 + j), A.h, iy, ty);
                    double a[6], da[6], b[6], db[6];
                    basis(ty, a); dbasis(ty, da);
                    basis(tx, b); dbasis(tx, db);
                    double f, gx, gy;
                    if (f_staged) {
                        const int wx = min(max(ix + B - 2 - fc0, 0), fww - 6), wy = min(max(iy + B - 2 - fr0, 0), fwh - 6);
                        f = contract_grad<double>(win + wy * fP + wx, fP, a, da, b, db, gx, gy);
                    } else {
                        f = contract_grad<double>(FC + (int64_t)(iy + B - 2) * cp + (ix + B - 2), cp, a, da, b, db, gx, gy);
                    }
                    pix1(j * T + t, (vm >> j) & 1u, f, gx, gy, dx, dy0 + j);
                }
            }
        }
    }
    warp_sums64<NVA>(acc, sm.red2[wid], lane);
    // ---- setup, pass 2 (ICGN): the Hessian's gradient moments, one pair of
    // gradient components at a time (15 sums live instead of 45) ------------
    if constexpr (!FAGN) {
#pragma unroll 1
        for (int pr = 0; pr < 3; pr++) {
            double mom[NMOM];
#pragma unroll
            for (int q = 0; q < NMOM; q++) mom[q] = 0.0;
            for (int t = tid; t < T; t += NT) {
                int dx, dy0;
                unpack_task(tasks[t], dx, dy0);
                double V[NB];
#pragma unroll
                for (int b = 0; b < NB; b++) V[b] = 0.0;
#pragma unroll
                for (int j = 0; j < kK; j++) {
                    const double2 g = RG[j * T + t];
                    const double gg = (pr == 2 ? g.y : g.x) * (pr == 0 ? g.x : g.y);
                    const double dyf = dy0 + j;
                    double pw = 1.0;
#pragma unroll
                    for (int b = 0; b < NB; b++) {
                        V[b] = fma(gg, pw, V[b]);
                        pw *= dyf;
                    }
                }
                double xp = 1.0;
#pragma unroll
                for (int a = 0; a < NB; a++) {
#pragma unroll
                    for (int b = 0; a + b < NB; b++) mom[mom_idx(a, b)] = fma(xp, V[b], mom[mom_idx(a, b)]);
                    xp *= (double)dx;
                }
            }
            warp_sums64<NMOM>(mom, sm.red2[wid] + NVA + pr * NMOM, lane);
        }
    }
    __syncthreads();
    constexpr int NV = FAGN ? NVA : NVA + 3 * NMOM;
    if (wid == 0) {
        for (int q = lane; q < NV; q += 32) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < NW; w++) t += sm.red2[w][q];
            sm.tot[q] = t;
        }
        __syncwarp();
        const int n = (int)(sm.tot[0] + 0.5);
        const double dn = (double)n;
        double ms = sm.tot[1] / (n > 0 ? dn : 1.0);  // mean of f - s
        double fm = shift + ms;
        if (n > 0 && !(sm.tot[2] - ms * sm.tot[1] > kLevelDigits * sm.tot[2])) {
            sums_about_mean<ORDER, FAGN>(RG, RF, RVM, tasks, T, fm, sm.tot, lane);
            ms = sm.tot[1] / dn;
            fm += ms;
        }
        const double dif = sm.tot[2] - ms * sm.tot[1], saa = dif < 0.0 ? 0.0 : dif;
        int st = GPV_OK;
        if (n == 0) st = GPV_EMPTY_MASK;
        else if (!(sqrt(saa / dn) > 1e-6 * fmax(1.0, fabs(fm)))) st = GPV_FEATURELESS;
        if (!FAGN && st == GPV_OK) {
            if (lane < M) {
                sm.A[lane] = sm.tot[4 + lane] - ms * sm.tot[4 + M + lane];  // sum SDI (f - f_m)
                sm.S[lane] = sm.tot[4 + M + lane];
            }
            for (int q = lane; q < 3 * NMOM; q += 32) sm.mom[q] = sm.tot[NVA + q];
            __syncwarp();
            const bool ok = hess_factor<ORDER>(sm.mom, sm.Hi, sm.L, sm.linv, sm.dsc, lane, kMinPivot);
            if (!ok) {
                moments_of_monomials<ORDER>(RG, RVM, tasks, T, sm.mom, lane);
                assemble_hessian<ORDER>(sm.mom, sm.L, lane);
                int g = 0;
                if (lane == 0) g = gj_inverse<M>(sm.L, sm.Hi);
                if (!__shfl_sync(0xffffffffu, g, 0)) st = GPV_SINGULAR_H;
            }
            if (lane == 0) sm.flag[3] = ok;
        }
        if (lane == 0) {
            sm.flag[0] = st;
            sm.misc[5] = fm;
            sm.misc[6] = saa;
            sm.misc[7] = sm.tot[3];
            sm.n_valid = n;
        }
    } else {
        int r0 = 0, c0 = 0, wh = 0, ww = 0, pitch = 0;
        const int4 ext = run_extent<ORDER>(sm.p, cx, cy, re, A.w, A.h);
        const bool ok = run_plan<16>(ext.x & ~kInside, ext.y, ext.z, ext.w, B, R.win_cap, r0, c0, wh, ww, pitch);
        if (ok) stage64<NT>(GC, cp, ch, r0, c0, wh, ww, pitch, win, 32);
        if (tid == 32) {
            sm.win_ok = ok;
            sm.win_r0 = r0; sm.win_c0 = c0; sm.win_h = wh; sm.win_w = ww; sm.win_p = pitch;
        }
    }
    __syncthreads();
    const int st0 = sm.flag[0], n = sm.n_valid;
    const double dn = (double)n, fm = sm.misc[5], saa = sm.misc[6], sssig = sm.misc[7];
    const double df = sqrt(saa);
    if (st0 != GPV_OK) {
        if (tid == 0) {
            write_failed(A, idx, d, M, st0, n, n ? fm : 0.0, n ? df : 0.0);
            if (st0 == GPV_SINGULAR_H) {
                A.out[idx].sssig = sssig;
                A.out[idx].sigma = sqrt(saa / dn);
            }
        }
        return;
    }
    // read by warp 0 only after the first iteration's barrier
    if (!FAGN && sm.flag[3]) hess_inverse_block<M, NT>(sm.L, sm.dsc, sm.Hi, tid);

    // ---- iterations ---------------------------------------------------------
    const double size = sqrt(dn);
    int iters = 0, status = GPV_OK;
    bool converged = false;
    double c_zncc = 0.0, c_znssd = 4.0, last_norm = 0.0;
    double cg = fm, rho = 1.0;              // ICGN: level of g, delta_f / delta_g of the last iteration
    double gm_last = 0.0, dg_last = 0.0;
    for (int it = 1; it <= A.max_iter; it++) {
        bool inside;
        {
            const int4 ext = run_extent<ORDER>(sm.p, cx, cy, re, A.w, A.h);
            inside = ext.x & kInside;
            const int xlo = ext.x & ~kInside, xhi = ext.y, ylo = ext.z, yhi = ext.w;
            if (!run_covers(sm, xlo, xhi, ylo, yhi, B)) {
                int r0, c0, wh, ww, pitch;
                const bool ok = run_plan<16>(xlo, xhi, ylo, yhi, B, R.win_cap, r0, c0, wh, ww, pitch);
                __syncthreads();  // nobody still reads the old window
                if (ok) stage64<NT>(GC, cp, ch, r0, c0, wh, ww, pitch, win, 0);
                if (tid == 0) {
                    sm.win_ok = ok;
                    sm.win_r0 = r0; sm.win_c0 = c0; sm.win_h = wh; sm.win_w = ww; sm.win_p = pitch;
                }
                __syncthreads();
            }
        }
        const bool staged = sm.win_ok != 0;
        const int gr0 = sm.win_r0, gc0 = sm.win_c0, gwh = sm.win_h, gww = sm.win_w, gP = sm.win_p;
        const double X0 = cx + sm.p[0], Y0 = cy + sm.p[1];
        const double bxd = floor(X0), byd = floor(Y0);
        const int wbx = (int)bxd, wby = (int)byd;
        const double ox = X0 == bxd ? 0.0 : X0 - bxd, oy = Y0 == byd ? 0.0 : Y0 - byd;  // (0 at an infinity too)
        double ux = 0., uy = 0., vx = 0., vy = 0., uxx = 0., uxy = 0., uyy = 0., vxx = 0., vxy = 0., vyy = 0.;
        if (ORDER >= 1) { ux = sm.p[2 % M]; vx = sm.p[3 % M]; uy = sm.p[4 % M]; vy = sm.p[5 % M]; }
        if (ORDER == 2) {
            uxx = 0.5 * sm.p[6 % M]; vxx = 0.5 * sm.p[7 % M]; uxy = sm.p[8 % M];
            vxy = sm.p[9 % M]; uyy = 0.5 * sm.p[10 % M]; vyy = 0.5 * sm.p[11 % M];
        }
        const int wy0 = wby + B - 2 - gr0, wx0 = wbx + B - 2 - gc0;
        const bool fast = staged && inside;
        // sweeps: 0 about the level of the iteration before; where that level or
        // rho costs digits, or the Hessian is so near singular that the
        // elimination inverted it, 1 the target's mean (about 0), 2 its spread about the
        // mean, 3 (ICGN) the sums with both
        for (int sweep = 0;; sweep++) {
        double sb = 0.0, sbb = 0.0, sab = 0.0, see = 0.0;
        double PB[FAGN ? 2 : M];
#pragma unroll
        for (int k = 0; k < (FAGN ? 2 : M); k++) PB[k] = 0.0;
        for (int t = tid; t < T; t += NT) {
            int dx, dy0;
            unpack_task(tasks[t], dx, dy0);
            const uint32_t vm = (uint32_t)RVM[t];
            const double dxf = dx;
            // position relative to (wbx + dx, wby + dy): A + B dy + C dy^2
            const double Ax = fma(fma(uxx, dxf, ux), dxf, ox), Ay = fma(fma(vxx, dxf, vx), dxf, oy);
            const double Bx = fma(uxy, dxf, uy), By = fma(vxy, dxf, vy);
            double m0x = 0.0, m0y = 0.0, m1x = 0.0, m1y = 0.0, m2x = 0.0, m2y = 0.0;
            auto take = [&](int j, double dyf, double g, double hx, double hy, double2 gf, double f) {
                const int sl = j * T + t;
                const bool in = (vm >> j) & 1u;
                if constexpr (FAGN) {
                    RT[sl] = g;
                    RH[sl] = make_double2(in ? hx : 0.0, in ? hy : 0.0);
                    const double b = in ? g - cg : 0.0;
                    sb += b;
                    sbb = fma(b, b, sbb);
                } else {
                    const double a = in ? f - fm : 0.0, b = in ? g - cg : 0.0;
                    const double e = fma(-rho, b, a);
                    sb += b;
                    sbb = fma(b, b, sbb);
                    sab = fma(a, b, sab);
                    see = fma(e, e, see);
                    const double gxb = gf.x * e, gyb = gf.y * e;
                    m0x += gxb;
                    m0y += gyb;
                    if (ORDER >= 1) { m1x = fma(gxb, dyf, m1x); m1y = fma(gyb, dyf, m1y); }
                    if (ORDER == 2) { const double d2 = dyf * dyf; m2x = fma(gxb, d2, m2x); m2y = fma(gyb, d2, m2y); }
                }
            };
            if (fast) {
                // no edge clamp can apply and the window covers every tap: the block rolls down the run
                double Rg[6][6];
                int fxp = 0, fyp = 0;
                const double *rbase = win + (dy0 + wy0) * gP + (dx + wx0);
#pragma unroll
                for (int j = 0; j < kK; j++) {
                    const double dyf = dy0 + j;
                    double2 gf = make_double2(0.0, 0.0);  // from L2: asked for at the sample's start
                    double f = 0.0;
                    if constexpr (!FAGN) {
                        gf = ld_pair(RG + j * T + t);
                        f = ld_one(RF + j * T + t);
                    }
                    double Lx = Ax, Ly = Ay;
                    if (ORDER == 1) { Lx = fma(Bx, dyf, Lx); Ly = fma(By, dyf, Ly); }
                    if (ORDER == 2) { Lx = fma(fma(uyy, dyf, Bx), dyf, Lx); Ly = fma(fma(vyy, dyf, By), dyf, Ly); }
                    const double flx = floor(Lx), fly = floor(Ly);
                    const int ix = (int)flx, iy = (int)fly;
                    const double tx = Lx - flx, ty = Ly - fly;
                    const double *rp = rbase + (j + iy) * gP + ix;
                    if (j == 0) {
#pragma unroll
                        for (int rr = 0; rr < 6; rr++)
#pragma unroll
                            for (int k = 0; k < 6; k++) Rg[rr][k] = rp[rr * gP + k];
                    } else {
                        if (ix != fxp || iy != fyp) {  // the block did not move down one row
#pragma unroll
                            for (int rr = 0; rr < 5; rr++)
#pragma unroll
                                for (int k = 0; k < 6; k++) Rg[(j + rr) % 6][k] = rp[rr * gP + k];
                        }
#pragma unroll
                        for (int k = 0; k < 6; k++) Rg[(j + 5) % 6][k] = rp[5 * gP + k];
                    }
                    fxp = ix;
                    fyp = iy;
                    double aw[6], bw[6], sr[6];
                    weights64(tx, bw);
#pragma unroll
                    for (int rr = 0; rr < 6; rr++) sr[rr] = dot6(Rg[(j + rr) % 6], bw);
                    weights64(ty, aw);
                    const double g = dot6(sr, aw);
                    double hx = 0.0, hy = 0.0;
                    if constexpr (FAGN) {
                        double w[6];
                        dbasis(ty, w);
                        hy = seq6(sr, w);
                        dbasis(tx, w);
#pragma unroll
                        for (int rr = 0; rr < 6; rr++) sr[rr] = seq6(Rg[(j + rr) % 6], w);
                        hx = seq6(sr, aw);
                    }
                    take(j, dyf, g, hx, hy, gf, f);
                }
            } else {
#pragma unroll 1
                for (int j = 0; j < kK; j++) {
                    const double dyf = dy0 + j;
                    const double Lx = fma(fma(uyy, dyf, Bx), dyf, Ax), Ly = fma(fma(vyy, dyf, By), dyf, Ay);
                    int ix, iy;
                    double tx, ty;
                    split_far(bxd + dxf, Lx, A.w, ix, tx);
                    split_far(byd + dyf, Ly, A.h, iy, ty);
                    double a[6], b[6], da[6], db[6], g, hx = 0.0, hy = 0.0;
                    basis(ty, a); basis(tx, b);
                    if constexpr (FAGN) { dbasis(ty, da); dbasis(tx, db); }
                    if (staged) {
                        const int wx = min(max(ix + B - 2 - gc0, 0), gww - 6), wy = min(max(iy + B - 2 - gr0, 0), gwh - 6);
                        if constexpr (FAGN) g = contract_grad<double>(win + wy * gP + wx, gP, a, da, b, db, hx, hy);
                        else g = contract<double>(win + wy * gP + wx, gP, a, b);
                    } else {
                        const C *q = GC + (int64_t)(iy + B - 2) * cp + (ix + B - 2);
                        if constexpr (FAGN) g = contract_grad<double>(q, cp, a, da, b, db, hx, hy);
                        else g = contract<double>(q, cp, a, b);
                    }
                    if constexpr (FAGN) take(j, dyf, g, hx, hy, make_double2(0.0, 0.0), 0.0);
                    else take(j, dyf, g, hx, hy, RG[j * T + t], RF[j * T + t]);
                }
            }
            if constexpr (!FAGN) {
                PB[0] += m0x;
                PB[1] += m0y;
                if (ORDER >= 1) {
                    PB[2 % M] = fma(dxf, m0x, PB[2 % M]); PB[3 % M] = fma(dxf, m0y, PB[3 % M]);
                    PB[4 % M] += m1x; PB[5 % M] += m1y;
                }
                if (ORDER == 2) {
                    const double h = 0.5 * dxf * dxf;
                    PB[6 % M] = fma(h, m0x, PB[6 % M]); PB[7 % M] = fma(h, m0y, PB[7 % M]);
                    PB[8 % M] = fma(dxf, m1x, PB[8 % M]); PB[9 % M] = fma(dxf, m1y, PB[9 % M]);
                    PB[10 % M] = fma(0.5, m2x, PB[10 % M]); PB[11 % M] = fma(0.5, m2y, PB[11 % M]);
                }
            }
        }
        double gmt, dg, t_fg;  // mean of b, delta_g, delta_f / delta_g
        if constexpr (FAGN) {
            // sweep 2: moments of the target's gradient about the warped centre, residual gradient, ZNSSD
            const double s0 = block_sum64<NT>(sb, sm), s1 = block_sum64<NT>(sbb, sm);
            gmt = s0 / dn;
            double dg2 = s1 - s0 * gmt;
            if (sweep == 2) {
                gmt = 0.0;
                dg2 = s1;
            } else if (sweep == 1 || !(dg2 > kLevelDigits * s1)) {  // the same for all threads
                cg = sweep ? cg + gmt : 0.0;
                continue;
            }
            dg = sqrt(dg2);
            t_fg = df / dg;
            const double gm = cg + gmt, ratio = dg / df, inv_df = 1.0 / df, inv_dg = 1.0 / dg;
            double mo[NMOM * 3], ac[M + 1];
#pragma unroll
            for (int q = 0; q < 3 * NMOM; q++) mo[q] = 0.0;
#pragma unroll
            for (int q = 0; q <= M; q++) ac[q] = 0.0;
            for (int t = tid; t < T; t += NT) {
                int dx, dy0;
                unpack_task(tasks[t], dx, dy0);
                const uint32_t vm = (uint32_t)RVM[t];
                const double dxf = dx;
                const double Ex = fma(fma(uxx, dxf, 1.0 + ux), dxf, 0.0), Ey = fma(fma(vxx, dxf, vx), dxf, 0.0);
                const double Bx = fma(uxy, dxf, uy), By = fma(vxy, dxf, 1.0 + vy);
#pragma unroll 1
                for (int j = 0; j < kK; j++) {
                    if (!((vm >> j) & 1u)) continue;
                    const int sl = j * T + t;
                    const double dyf = dy0 + j;
                    // offsets from the warped centre
                    const double X = fma(fma(uyy, dyf, Bx), dyf, Ex), Y = fma(fma(vyy, dyf, By), dyf, Ey);
                    const double2 h = RH[sl];
                    const double a = RF[sl] - fm, b = RT[sl] - gm;
                    const double z = fma(a, inv_df, -(b * inv_dg));
                    ac[M] = fma(z, z, ac[M]);
                    const double res = fma(a, ratio, -b);
#pragma unroll
                    for (int mu = 0; mu < NMU; mu++) {
                        const double w = mu_val<double>(mu, X, Y) * res;
                        ac[2 * mu] = fma(h.x, w, ac[2 * mu]);
                        ac[2 * mu + 1] = fma(h.y, w, ac[2 * mu + 1]);
                    }
                    const double hh[3] = {h.x * h.x, h.x * h.y, h.y * h.y};
                    double xp = 1.0;
#pragma unroll
                    for (int ea = 0; ea < NB; ea++) {
                        double mono = xp;
#pragma unroll
                        for (int eb = 0; ea + eb < NB; eb++) {
#pragma unroll
                            for (int q = 0; q < 3; q++)
                                mo[q * NMOM + mom_idx(ea, eb)] = fma(hh[q], mono, mo[q * NMOM + mom_idx(ea, eb)]);
                            mono *= Y;
                        }
                        xp *= X;
                    }
                }
            }
            warp_sums64<M + 1>(ac, sm.red2[wid], lane);
            warp_sums64<3 * NMOM>(mo, sm.red2[wid] + M + 1, lane);
        } else {
            constexpr int KR = 4 + M;
            double v[KR];
            v[0] = sb; v[1] = sbb; v[2] = sab; v[3] = see;
#pragma unroll
            for (int j = 0; j < M; j++) v[4 + j] = PB[j];
            warp_sum_many<KR>(v, sm.red[wid], lane);
        }
        __syncthreads();
        if (wid == 0) {
            double dpj = 0.0, znssd;
            bool ok = true, again = false;
            if constexpr (FAGN) {
                for (int q = lane; q < M + 1 + 3 * NMOM; q += 32) {
                    double t = 0.0;
#pragma unroll
                    for (int w = 0; w < NW; w++) t += sm.red2[w][q];
                    if (q <= M) sm.tot[q] = t;
                    else sm.mom[q - M - 1] = t;
                }
                __syncwarp();
                znssd = sm.tot[M];
                // dp = H^-1 grad by the factor's inverse: D L^-T (L^-1 (D grad))
                if (hess_factor<ORDER>(sm.mom, sm.Hi, sm.L, sm.linv, sm.dsc, lane, kMinPivot)) {
                    double y = 0.0;
                    if (lane < M) {
#pragma unroll
                        for (int k = 0; k < M; k++) y = fma(sm.L[lane * M + k], sm.dsc[k] * sm.tot[k], y);
                        sm.grad[lane] = y;
                    }
                    __syncwarp();
                    if (lane < M) {
#pragma unroll
                        for (int k = 0; k < M; k++) dpj = fma(sm.L[k * M + lane], sm.grad[k], dpj);
                        dpj *= sm.dsc[lane];
                    }
                } else {
                    assemble_hessian<ORDER>(sm.mom, sm.L, lane);
                    int g = 0;
                    if (lane == 0) g = gj_inverse<M>(sm.L, sm.Hi);
                    ok = __shfl_sync(0xffffffffu, g, 0) != 0;
                    __syncwarp();  // lane 0's inverse is read below (a shuffle orders no memory)
                    if (ok && lane < M)
                        for (int k = 0; k < M; k++) dpj = fma(sm.Hi[lane * M + k], sm.tot[k], dpj);
                }
            } else {
                double tl = 0.0;
                if (lane < 4 + M) {
#pragma unroll
                    for (int w = 0; w < NW; w++) tl += sm.red[w][lane];
                }
                const double tb = __shfl_sync(0xffffffffu, tl, 0), tbb = __shfl_sync(0xffffffffu, tl, 1);
                const double tab = __shfl_sync(0xffffffffu, tl, 2), tee = __shfl_sync(0xffffffffu, tl, 3);
                gmt = tb / dn;
                double dg2 = tbb - tb * gmt;
                if (sweep == 0) {
                    again = !(dg2 > kLevelDigits * tbb && rho * rho * dg2 <= kScaleDigits * saa) || !sm.flag[3];
                } else {
                    again = sweep < 3;
                    if (sweep > 1) {  // about the mean itself
                        gmt = 0.0;
                        dg2 = tbb;
                    }
                }
                dg = sqrt(dg2);
                t_fg = df / dg;
                // sum (e - k b + t d)^2 with sum e = -rho sum b (sum a = 0) and sum e b = sum a b - rho sum b^2
                const double k = t_fg - rho, td = t_fg * gmt;
                const double srr = sweep == 3 ? tee  // rho is t
                                              : tee + k * (k * tbb - 2.0 * (tab - rho * tbb)) - 2.0 * td * (rho * tb + k * tb) + dn * td * td;
                znssd = (srr < 0.0 ? 0.0 : srr) / saa;  // a NaN (delta_g = 0) stays one
                const double ej = __shfl_down_sync(0xffffffffu, tl, 4);
                if (lane < M) {
                    const double corr = k == 0.0 ? 0.0 : k * ((sm.A[lane] - ej) / rho);
                    sm.grad[lane] = ej - corr + td * sm.S[lane];
                }
                __syncwarp();
                if (lane < M) {
                    double a0 = 0.0, a1 = 0.0;
#pragma unroll
                    for (int q = 0; q < M; q += 2) {
                        a0 = fma(sm.Hi[lane * M + q], sm.grad[q], a0);
                        a1 = fma(sm.Hi[lane * M + q + 1], sm.grad[q + 1], a1);
                    }
                    dpj = -(a0 + a1);
                }
            }
            if (lane < M && !again) {
                sm.dp[lane] = dpj;
                sm.pprev[lane] = sm.p[lane];
            }
            __syncwarp();
            if (lane == 0 && again) {
                sm.flag[1] = 2;
                sm.misc[2] = gmt;
                sm.misc[9] = t_fg;
            } else if (lane == 0) {
                double dpl[12], pl[12];
#pragma unroll
                for (int k = 0; k < 12; k++) {
                    dpl[k] = sm.dp[k % M];
                    pl[k] = sm.p[k % M];
                }
                if constexpr (FAGN) {
                    if (ok) {
#pragma unroll
                        for (int k = 0; k < M; k++) sm.p[k] = pl[k] + dpl[k];
                    }
                } else {
                    double pn[12];
                    if (ORDER == 0) {
                        pn[0] = pl[0] - dpl[0];
                        pn[1] = pl[1] - dpl[1];
                    } else if (ORDER == 1) {
                        ok = compose1(pl, dpl, pn);
                    } else {
                        ok = compose2_any(pl, dpl, pn, sm.red2[0]);
                    }
                    if (ok) {
#pragma unroll
                        for (int k = 0; k < M; k++) sm.p[k] = pn[k];
                    }
                }
                sm.flag[1] = ok;
                sm.misc[1] = conv_norm<M>(dpl, size);
                sm.misc[2] = gmt;
                sm.misc[3] = dg;
                sm.misc[4] = znssd;
                sm.misc[9] = t_fg;
            }
        }
        __syncthreads();
        if (FAGN || sm.flag[1] < 2) break;
        if (sweep == 0) cg = 0.0;
        else if (sweep == 1) cg = sm.misc[2];
        else rho = sm.misc[9];
        }
        gm_last = cg + sm.misc[2];
        dg_last = sm.misc[3];
        if (!sm.flag[1]) {  // p keeps the last valid warp
            status = FAGN ? GPV_SINGULAR_H : GPV_SINGULAR_WDELTA;
            break;
        }
        const double nrm = sm.misc[1];
        c_znssd = sm.misc[4];
        c_zncc = 1.0 - c_znssd / 2.0;
        iters = it;
        last_norm = nrm;
        if (tid == 0) write_history(A, idx, it, nrm, c_zncc, c_znssd);
        if (!isfinite(nrm)) { status = GPV_NONFINITE; break; }
        if (nrm < A.max_norm) { converged = true; break; }
        // the next iteration's level and scale
        cg = gm_last;
        rho = sm.misc[9];
    }

    // ---- eta diagnostic at the last sampled warp (optional) -----------------
    double eu = 0.0, ev = 0.0;
    const bool want_eta = ETA && iters > 0 && status == GPV_OK;
    if (ETA && want_eta) {
        const double *pp = sm.pprev;
        const double X0 = cx + pp[0], Y0 = cy + pp[1];
        const double bxd = floor(X0), byd = floor(Y0);
        // this thread's template pixels; the first walk (FIRST) samples g again where the solve kept none
        auto each = [&](auto first, auto fn) {
#pragma unroll 1
            for (int t = tid; t < T; t += NT) {
                int dxi, dy0;
                unpack_task(tasks[t], dxi, dy0);
                const int vm = RVM[t];
#pragma unroll 1
                for (int j = 0; j < kK; j++) {
                    if (!((vm >> j) & 1)) continue;
                    const int sl = j * T + t;
                    const double dx = dxi, dy = dy0 + j;
                    if constexpr (!FAGN && decltype(first)::value) {
                        double lx = X0 == bxd ? 0.0 : X0 - bxd, ly = Y0 == byd ? 0.0 : Y0 - byd;
                        if (ORDER >= 1) {
                            lx += pp[2 % M] * dx + pp[4 % M] * dy;
                            ly += pp[3 % M] * dx + pp[5 % M] * dy;
                        }
                        if (ORDER == 2) {
                            lx += 0.5 * pp[6 % M] * dx * dx + pp[8 % M] * dx * dy + 0.5 * pp[10 % M] * dy * dy;
                            ly += 0.5 * pp[7 % M] * dx * dx + pp[9 % M] * dx * dy + 0.5 * pp[11 % M] * dy * dy;
                        }
                        int ix, iy;
                        double tx, ty;
                        split_far(bxd + dx, lx, A.w, ix, tx);
                        split_far(byd + dy, ly, A.h, iy, ty);
                        double a[6], b[6];
                        basis(ty, a);
                        basis(tx, b);
                        RT[sl] = contract<double>(GC + (int64_t)(iy + B - 2) * cp + (ix + B - 2), cp, a, b);
                    }
                    const double2 q = RG[sl];
                    fn(RF[sl] - fm, q.x, q.y, RT[sl] - gm_last, dx, dy);
                }
            }
        };
        auto red = [&](auto &v) { run_block_sums<NT>(v, sm.red2, sm.tot); };
        eta_two_pass<ORDER>(dn, df, dg_last, each, red, eu, ev);
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
        o->sssig = sssig;
        o->sigma = sqrt(saa / dn);
        o->iterations = iters;
        o->converged = converged;
        o->quality_ok = converged && c_zncc >= A.tolerance;
        o->status = status;
        o->n_px = n;
        o->has_eta = want_eta;
        o->texture = 0;
        o->reserved = 0;
    }
}

// Blocks take subsets of their segment from the queue.  Three blocks of 128
// threads per SM (168 registers); the second-order ICGN sweep, whose sums alone
// take 70 registers, does better with two at 255 and no spills (2.40 against
// 2.55 ms on 8,836 subsets of radius 30; first order 1.95 against 1.81).
template <int ORDER, int NT, bool FAGN, typename C, bool ETA>
__global__ void __launch_bounds__(NT, NT == 128 ? (ORDER == 2 && !FAGN ? 2 : 3) : 1) icgn_runs64(RunArgs R) {
    extern __shared__ double2 win2[];
    __shared__ Smem64<NT / 32> sm;
    const KArgs &A = R.k;
    const int start = R.seg[0], count = R.seg[1];
    double *base = reinterpret_cast<double *>(A.scratch) + (int64_t)blockIdx.x * A.scratch_stride;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) sm.item = atomicAdd(R.queue, 1);
        __syncthreads();
        const int item = sm.item;
        if (item >= count) break;
        const int idx = A.order[start + item];
        const gpv_subset_desc d = A.desc[idx];
        run64_subset<ORDER, NT, FAGN, C, ETA>(R, idx, d, base, reinterpret_cast<double *>(win2), sm);
    }
}

template <int NT, bool FAGN, typename C, bool ETA>
const void *kernel64_t(int order) {
    return order == 2 ? (const void *)icgn_runs64<2, NT, FAGN, C, ETA>
                      : (order == 1 ? (const void *)icgn_runs64<1, NT, FAGN, C, ETA>
                                    : (const void *)icgn_runs64<0, NT, FAGN, C, ETA>);
}

template <int NT, bool ETA>
const void *kernel64_nt(int order, bool fagn, bool c64) {
    if (!fagn) return kernel64_t<NT, false, double, ETA>(order);
    return c64 ? kernel64_t<NT, true, double, ETA>(order) : kernel64_t<NT, true, float, ETA>(order);
}

}  // namespace

// Window capacity (doubles): as run_window_cap, at the FP64 pitch.
int run64_window_cap(int rmax) {
    const int e = std::max(rmax, kK - 1 - rmax);
    const int rw = (int)std::ceil(1.06 * e) + 2;
    const int side = 2 * rw + 6 + 2 * kRunMargin + 4;
    return side * run_pitch<16>(side);
}

// Scratch doubles per block for nslot record slots (run_scratch_floats gives
// the slots): 4 per slot (FAGN 6), and the runs' pixel bits.
int64_t run64_scratch_doubles(int nslot, bool fagn) {
    return (fagn ? 6 : 4) * (int64_t)nslot + nslot / (2 * kK) + 16;
}

const void *run64_kernel(int order, int nt, bool fagn, bool c64, bool eta) {
    if (eta) return nt == 256 ? kernel64_nt<256, true>(order, fagn, c64) : kernel64_nt<128, true>(order, fagn, c64);
    return nt == 256 ? kernel64_nt<256, false>(order, fagn, c64) : kernel64_nt<128, false>(order, fagn, c64);
}

int run64_launch(gpv_context *ctx, const void *fn, int nt, int blocks, size_t smem, cudaStream_t s, const KArgs &k,
                 const int32_t *seg, int *queue, int win_cap, int nslot) {
    RunArgs R;
    R.k = k;
    run_tables(ctx, R);
    R.seg = seg;
    R.queue = queue;
    R.win_cap = win_cap;
    R.nslot = nslot;
    R.slot_mask = nullptr;
    R.slots_per_sm = R.n_mask = 0;
    void *args[] = {&R};
    GPV_CUDA_TRY(cudaLaunchKernel(fn, dim3((unsigned)blocks), dim3((unsigned)nt), args, smem, s));
    return GPV_SUCCESS;
}

}  // namespace gpv
