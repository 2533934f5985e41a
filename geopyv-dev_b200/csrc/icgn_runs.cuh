// icgn_runs.cuh -- pieces shared by the run-layout solves (icgn_runs.cu in
// mixed precision, icgn_runs64.cu in FP64): the launch arguments, the window
// planning, the Hessian's factor and inverse.
#pragma once
#include <type_traits>

#include "icgn_common.cuh"
#include "run_window.h"

namespace gpv {
namespace {

struct RunArgs {
    KArgs k;
    const int2 *tasks;        // run tables
    const int32_t *task_off;  // [radius]: first task of the radius
    const int32_t *task_n;    // [radius]: tasks of the radius
    const int32_t *seg;       // [start, count] of this segment in k.order
    int *queue;               // this launch's work-queue counter
    int win_cap;              // floats of dynamic shared memory for a window
    int nslot;                // record slots per block (tasks x K of the segment's largest radius, rounded)
    // one block per subset (slot_mask != nullptr): a block claims one of the
    // slots_per_sm scratch slots of the SM it starts on (a bit of
    // slot_mask[smid], n_mask words) and frees it when the subset is done
    uint32_t *slot_mask;
    int slots_per_sm, n_mask;
};

// Scratch floats of a block without the rigid template's part: float4 records,
// the diagnostic's samples, the runs' pixel bits (nslot / kRunK runs at most).
__host__ __device__ __forceinline__ int64_t run_plain_floats(int nslot) {
    return 5 * (int64_t)nslot + (nslot / kRunK + 31) / 32 * 32;
}

// The context's run tables (ensure_run_tables).
inline void run_tables(const gpv_context *ctx, RunArgs &R) {
    const int32_t *t = static_cast<const int32_t *>(ctx->run_tab.ptr);
    const int R1 = ctx->run_table_radius + 1;
    R.task_off = t;
    R.task_n = t + R1;
    R.tasks = reinterpret_cast<const int2 *>(t + 2 * R1);
}

template <class S>
__device__ __forceinline__ bool run_covers(const S &sm, int xlo, int xhi, int ylo, int yhi, int border) {
    if (!sm.win_ok) return false;
    return xlo + border - 2 >= sm.win_c0 && xhi + border + 3 < sm.win_c0 + sm.win_w && ylo + border - 2 >= sm.win_r0 &&
           yhi + border + 3 < sm.win_r0 + sm.win_h;
}

// Pixel extent (image pixels, clamped) {xlo, xhi, ylo, yhi} of the square
// [-e, e]^2 of a subset centred at (cx, cy) under the warp p, conservatively;
// xlo carries kInside when the extent with a one-pixel margin lies in the
// image (no sample meets the edge clamp).  A warp that is not finite gives the
// whole image.
constexpr int kInside = 1 << 30;
template <int ORDER>
__device__ __forceinline__ int4 run_extent(const double *p, double cx, double cy, int e, int w, int h) {
    __builtin_assume(__isShared(p));
    double ex = e, ey = e;
    if (ORDER >= 1) {
        ex = e * (fabs(1.0 + p[2]) + fabs(p[4]));
        ey = e * (fabs(p[3]) + fabs(1.0 + p[5]));
    }
    if (ORDER == 2) {
        const double rr = 0.5 * (double)e * e;
        ex += rr * (fabs(p[6 % 12]) + 2.0 * fabs(p[8 % 12]) + fabs(p[10 % 12]));
        ey += rr * (fabs(p[7 % 12]) + 2.0 * fabs(p[9 % 12]) + fabs(p[11 % 12]));
    }
    const double X0 = cx + p[0], Y0 = cy + p[1];
    if (!isfinite(fabs(X0) + ex + fabs(Y0) + ey)) return make_int4(0, w - 1, 0, h - 1);
    // floors, saturated to int and kept clear of its ends
    constexpr int kEnd = 1 << 29;
    const int a = max(min(__double2int_rd(X0 - ex), kEnd), -kEnd) - 1, b = max(min(__double2int_rd(X0 + ex), kEnd), -kEnd) + 1;
    const int c = max(min(__double2int_rd(Y0 - ey), kEnd), -kEnd) - 1, d = max(min(__double2int_rd(Y0 + ey), kEnd), -kEnd) + 1;
    const bool inside = a >= 0 && b <= w - 1 && c >= 0 && d <= h - 1;
    return make_int4(max(min(a, w - 1), 0) | (inside ? kInside : 0), max(min(b, w - 1), 0), max(min(c, h - 1), 0),
                     max(min(d, h - 1), 0));
}

// The Cholesky factor of the Jacobi-scaled SPD Hessian and the factor's
// inverse, by one warp: D H D = L L^T with D = diag(1 / sqrt(H_jj)), so
// H^-1 = D L^-T L^-1 D.  Lane i < M holds row i in registers, shifted down one
// place per step so that the current column is always its first entry: the
// steps then are passes of one rolled loop (registers cannot be indexed by the
// step).  Unrolled, this took 21 KB of instructions of the second-order solve
// for a stretch run once per subset, and instruction fetch (32 KB of cache per
// SM, the solve's blocks in different phases) bounded the solve.
// The rows are built from the gradient moments without the monomials'
// factors c_j (1 or 1/2), which the scaling takes out again: H_jk = c_j c_k
// sum g_p g_q dx^a dy^b.  Each pivot takes one reciprocal square root.  Lane c
// then solves L x = e_c for column c of L^-1, in the same shifted form.
// Lw: M * M + 16 scratch (columns of L); Li: L^-1, row-major, zeros above the
// diagonal; linv: M scratch; dsc: 1 / sqrt(H_jj).  False (warp-uniform) when
// a pivot is not above min_piv (the scaled diagonal is 1) or not finite: a singular Hessian.
template <int ORDER>
__device__ __forceinline__ bool hess_factor(const double *mom, double *Lw, double *Li, double *linv, double *dsc, int lane,
                                            double min_piv = 0.0) {
    using O = Ord<ORDER>;
    constexpr int M = O::M;
    constexpr unsigned kAll = 0xffffffffu;
    __builtin_assume(__isShared(mom));
    __builtin_assume(__isShared(Lw));
    __builtin_assume(__isShared(Li));
    __builtin_assume(__isShared(linv));
    __builtin_assume(__isShared(dsc));
    const int li = lane < M ? lane : 0;  // lanes >= M shadow row 0; their results are never read
    const int mi = li >> 1, ci = li & 1, ai = mu_a(mi), bi = mu_b(mi);
    double h[M];
#pragma unroll
    for (int k = 0; k < M; k++) h[k] = mom[(ci + (k & 1)) * O::NMOM + mom_idx(ai + mu_a(k >> 1), bi + mu_b(k >> 1))];
    const double dii = mom[(2 * ci) * O::NMOM + mom_idx(2 * ai, 2 * bi)];  // h[li]
    if (__any_sync(kAll, !(dii > 0.0) || !isfinite(dii))) return false;
    const double si = rsqrt(dii);
#pragma unroll
    for (int j = 0; j < M; j++) h[j] *= si * __shfl_sync(kAll, si, j);
#pragma unroll 1
    for (int k = 0; k < M; k++) {
        const double piv = __shfl_sync(kAll, h[0], k);
        if (!(piv > min_piv) || !isfinite(piv)) return false;  // uniform: every lane has lane k's value
        const double rk = rsqrt(piv);
        const double lik = li > k ? h[0] * rk : (li == k ? piv * rk : 0.0);
        if (lane < M) Lw[k * M + lane] = lik;
        if (lane == k) linv[k] = rk;
#pragma unroll
        for (int j = 1; j < M; j++) h[j - 1] = fma(-lik, __shfl_sync(kAll, lik, (k + j) & 31), h[j]);
    }
    __syncwarp();
    double x[M];
#pragma unroll
    for (int i = 0; i < M; i++) x[i] = (i == lane) ? 1.0 : 0.0;
#pragma unroll 1
    for (int k = 0; k < M; k++) {
        const double xk = x[0] * linv[k];
        if (lane < M) Li[k * M + lane] = xk;
        const double *col = Lw + k * M + k;  // entries past the column's end only reach values never used
#pragma unroll
        for (int j = 1; j < M; j++) x[j - 1] = fma(-col[j], xk, x[j]);
    }
    if (lane < M) dsc[lane] = (mi == 3 || mi == 5) ? si + si : si;
    __syncwarp();
    return true;
}

// H^-1 = D L^-T L^-1 D from hess_factor's L^-1 (Lm) and D (dsc), by
// the whole block between two barriers (no warp waits on another's serial
// work here): entry (i, j) is s_i s_j times the dot product of columns i
// and j of L^-1.
template <int M, int NT>
__device__ __forceinline__ void hess_inverse_block(const double *Lm, const double *dsc, double *Hi, int tid) {
#pragma unroll 1
    for (int e = tid; e < M * M; e += NT) {
        const int i = e / M, j = e - (e / M) * M;
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < M; k++) acc = fma(Lm[k * M + i], Lm[k * M + j], acc);
        Hi[e] = dsc[i] * dsc[j] * acc;
    }
}

__device__ __forceinline__ void unpack_task(int2 tk, int &dx, int &dy0) {
    dx = (int)(short)(tk.x & 0xffff);
    dy0 = tk.x >> 16;
}

// Warp sums of KV values into dst[0..KV), 16 at a time.
template <int KV, int C = 0>
__device__ __forceinline__ void warp_sums64(const double (&a)[KV], double *dst, int lane) {
    if constexpr (C < KV) {
        constexpr int N = (KV - C) < 16 ? (KV - C) : 16;
        double v[N];
#pragma unroll
        for (int j = 0; j < N; j++) v[j] = a[C + j];
        warp_sum_many<N>(v, dst + C, lane);
        warp_sums64<KV, C + N>(a, dst, lane);
    }
}


// Block sums of N per-thread values in place, every thread receiving the
// totals: warp sums in red2, one thread per value adding them into out.
template <int NT, int N, int W>
__device__ __forceinline__ void run_block_sums(double (&v)[N], double (&red2)[NT / 32][W], double *out) {
    static_assert(N <= W && N <= NT, "one thread per value");
    warp_sums64<N>(v, red2[threadIdx.x >> 5], threadIdx.x & 31);
    __syncthreads();
    if (threadIdx.x < N) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < NT / 32; w++) t += red2[w][threadIdx.x];
        out[threadIdx.x] = t;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < N; q++) v[q] = out[q];
}

// Omitted-mode diagnostic (src/subset.rs:698-820) in two walks over a
// block's pixels: the moments of the residual and of the gradients, then for
// every (component, mode) the sums of the raw mode, its square and its product
// with the residual together (6 K sums and one reduction, where a walk and
// three block sums per (component, mode) took 70 us of a single subset's
// 111 us solve).  each(first, fn) calls fn(f - f_m, gx, gy, g - g_m, dx, dy)
// for this thread's pixels; reduce(v) sums an array over the block.
template <int ORDER, class Each, class Reduce>
__device__ __forceinline__ void eta_two_pass(double n, double df, double dg, Each each, Reduce reduce, double &eu,
                                             double &ev) {
    constexpr int K = ORDER + 2;
    const double idf = 1.0 / df, idg = 1.0 / dg;
    double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    each(std::true_type(), [&](double a, double gx, double gy, double b, double, double) {
        s[0] += a * idf - b * idg;
        s[1] += gx; s[2] += gx * gx;
        s[3] += gy; s[4] += gy * gy;
    });
    reduce(s);
    const double eb = s[0] / n, mx = s[1] / n, my = s[3] / n;
    const double ix = rsqrt(fmax(s[2] / n - mx * mx, 1e-18)), iy = rsqrt(fmax(s[4] / n - my * my, 1e-18));
    double t[6 * K];
#pragma unroll
    for (int q = 0; q < 6 * K; q++) t[q] = 0.0;
    each(std::false_type(), [&](double a, double gx, double gy, double b, double dx, double dy) {
        const double e = a * idf - b * idg, zx = (gx - mx) * ix, zy = (gy - my) * iy;
#pragma unroll
        for (int k = 0; k < K; k++) {  // modes dx^(ORDER+1-k) dy^k
            double md = 1.0;
#pragma unroll
            for (int q = 0; q < K - 1; q++) md *= q < K - 1 - k ? dx : dy;
            const double rx = zx * md, ry = zy * md;
            t[6 * k] += rx; t[6 * k + 1] += rx * rx; t[6 * k + 2] += rx * e;
            t[6 * k + 3] += ry; t[6 * k + 4] += ry * ry; t[6 * k + 5] += ry * e;
        }
    });
    reduce(t);
    double eta[2] = {0.0, 0.0};
#pragma unroll 1
    for (int c = 0; c < 2; c++) {
        double ss = 0.0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const double a1 = c ? t[6 * k + 3] : t[6 * k], a2 = c ? t[6 * k + 4] : t[6 * k + 1],
                         a3 = c ? t[6 * k + 5] : t[6 * k + 2];
            const double mean = a1 / n, var = fmax(a2 / n - mean * mean, 1e-18);
            const double pr = (a3 - eb * a1) * rsqrt(var) / n;
            ss += pr * pr;
        }
        eta[c] = sqrt(ss);
    }
    eu = eta[0];
    ev = eta[1];
}

}  // namespace
}  // namespace gpv
