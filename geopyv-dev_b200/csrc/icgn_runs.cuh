// icgn_runs.cuh -- pieces shared by the run-layout solves (icgn_runs.cu in
// mixed precision, icgn_runs64.cu in FP64): the launch arguments, the window
// planning, the Hessian's factor and inverse.
#pragma once
#include "icgn_common.cuh"

namespace gpv {
namespace {

constexpr int kRunMargin = 4;

struct RunArgs {
    KArgs k;
    const int2 *tasks;        // task tables of this launch's run length K
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

// Window row pitch in elements: a multiple of 4 (16-byte rows for cp.async)
// that is not a multiple of BANKS, the elements one row of shared-memory banks
// holds (32 floats, 16 doubles), so two bands' rows read by one warp start on
// different banks.  Lanes of a warp read consecutive columns of one row.
template <int BANKS>
__host__ __device__ __forceinline__ int run_pitch(int ww) {
    const int p = (ww + 3) & ~3;
    return (p & (BANKS - 1)) ? p : p + 4;
}

// A window covering pixel indices [xlo, xhi] x [ylo, yhi] (clamped to the
// image) plus the taps and kRunMargin; false if it does not fit in cap
// elements (the margin is dropped when the window with it does not fit).
template <int BANKS>
__device__ __forceinline__ bool run_plan(int xlo, int xhi, int ylo, int yhi, int border, int cap, int &r0, int &c0,
                                         int &wh, int &ww, int &pitch) {
    for (int m = kRunMargin; m >= 0; m -= kRunMargin) {
        const int clo = xlo + border - 2 - m, chi = xhi + border + 3 + m;
        c0 = clo >= 0 ? (clo & ~3) : -(((-clo) + 3) & ~3);
        ww = ((chi + 1 - c0) + 3) & ~3;
        pitch = run_pitch<BANKS>(ww);
        r0 = ylo + border - 2 - m;
        wh = yhi + border + 3 + m + 1 - r0;
        if (pitch * wh <= cap) return true;
        if (m == 0) break;
    }
    return false;
}

template <class S>
__device__ __forceinline__ bool run_covers(const S &sm, int xlo, int xhi, int ylo, int yhi, int border) {
    if (!sm.win_ok) return false;
    return xlo + border - 2 >= sm.win_c0 && xhi + border + 3 < sm.win_c0 + sm.win_w && ylo + border - 2 >= sm.win_r0 &&
           yhi + border + 3 < sm.win_r0 + sm.win_h;
}

// Pixel extent (image pixels, clamped) of the square [-e, e]^2 of a subset
// centred at (cx, cy) under the warp p, conservatively; *inside: the extent
// with a one-pixel margin lies in the image (no sample meets the edge clamp).
template <int ORDER>
__device__ void run_extent(const double *p, double cx, double cy, int e, int w, int h, int &xlo, int &xhi, int &ylo,
                           int &yhi, bool *inside) {
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
    const double a = floor(X0 - ex) - 1.0, b = floor(X0 + ex) + 1.0, c = floor(Y0 - ey) - 1.0, d = floor(Y0 + ey) + 1.0;
    if (!(isfinite(a) && isfinite(b) && isfinite(c) && isfinite(d))) {
        xlo = 0; xhi = w - 1; ylo = 0; yhi = h - 1;  // plans a window that cannot fit: global path
        *inside = false;
        return;
    }
    *inside = a >= 0.0 && b <= (double)(w - 1) && c >= 0.0 && d <= (double)(h - 1);
    xlo = (int)fmax(0.0, fmin(a, (double)(w - 1)));
    xhi = (int)fmax(0.0, fmin(b, (double)(w - 1)));
    ylo = (int)fmax(0.0, fmin(c, (double)(h - 1)));
    yhi = (int)fmax(0.0, fmin(d, (double)(h - 1)));
}

// The Cholesky factor of the Jacobi-scaled SPD Hessian and the factor's
// inverse, by one warp in registers: D H D = L L^T with D = diag(1 /
// sqrt(H_jj)), so H^-1 = D L^-T L^-1 D.  Lane i < M builds row i of H from the gradient
// moments (H_jk = c_j c_k sum g_p g_q dx^a dy^b, the entries assemble_hessian
// gives) and keeps it in registers; the pivot and the column entries each
// step needs travel by shuffle.  Each pivot takes one reciprocal square root
// (1 / L_kk, and L_kk = pivot x that), not a square root and a division:
// the serial chain of a lone warp is what this stretch costs.  Lane c then
// solves L x = e_c for column c of L^-1 (rows of L read from Lm, M*M shared
// scratch), which then holds L^-1 (zeros above the diagonal), and lane i
// stores s_i = 1 / sqrt(H_ii) in dsc; hess_inverse_block forms H^-1 from
// them.  False (warp-uniform) when a pivot is not positive or not finite:
// a singular Hessian.
template <int ORDER>
__device__ bool hess_factor_regs(const double *mom, double *Lm, double *linv, double *dsc, int lane) {
    using O = Ord<ORDER>;
    constexpr int M = O::M;
    constexpr unsigned kAll = 0xffffffffu;
    const int li = lane < M ? lane : 0;  // lanes >= M shadow row 0; their results are never read
    const int mi = li >> 1, ci = li & 1, ai = mu_a(mi), bi = mu_b(mi);
    const double cci = mu_c(mi);
    double h[M];
#pragma unroll
    for (int k = 0; k < M; k++) {
        const int mk = k >> 1, ck = k & 1;
        h[k] = cci * mu_c(mk) * mom[(ci + ck) * O::NMOM + mom_idx(ai + mu_a(mk), bi + mu_b(mk))];
    }
    const double dii = cci * cci * mom[(2 * ci) * O::NMOM + mom_idx(2 * ai, 2 * bi)];  // h[li]
    if (__any_sync(kAll, !(dii > 0.0) || !isfinite(dii))) return false;
    const double si = rsqrt(dii);
#pragma unroll
    for (int j = 0; j < M; j++) {
        const double sj = __shfl_sync(kAll, si, j);
        h[j] *= si * sj;
    }
    // 1 / L_kk into linv (shared, M doubles) by lane k
#pragma unroll
    for (int k = 0; k < M; k++) {
        const double piv = __shfl_sync(kAll, h[k], k);
        if (!(piv > 0.0) || !isfinite(piv)) return false;  // uniform: every lane has lane k's value
        const double rk = rsqrt(piv);
        const double lkk = piv * rk;
        if (lane == k) linv[k] = rk;
        h[k] = li > k ? h[k] * rk : (li == k ? lkk : h[k]);
#pragma unroll
        for (int j = k + 1; j < M; j++) {
            const double ljk = __shfl_sync(kAll, h[k], j);
            if (li >= j) h[j] = fma(-h[k], ljk, h[j]);
        }
    }
    if (lane < M) {
#pragma unroll
        for (int j = 0; j < M; j++) Lm[lane * M + j] = j <= lane ? h[j] : 0.0;
    }
    __syncwarp();
    // column c = lane of L^-1 by forward substitution (zero above the
    // diagonal), right-looking: each x_k, once known, updates every later
    // row at once, so the dependent chain is M steps, not M (M - 1) / 2
    double x[M];
#pragma unroll
    for (int i = 0; i < M; i++) x[i] = (i == lane) ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < M; k++) {
        x[k] = (k >= lane) ? x[k] * linv[k] : 0.0;
#pragma unroll
        for (int i = k + 1; i < M; i++) x[i] = fma(-Lm[i * M + k], x[k], x[i]);
    }
    __syncwarp();
    if (lane < M) {
#pragma unroll
        for (int i = 0; i < M; i++) Lm[i * M + lane] = x[i];  // Lm now holds L^-1 (lower)
    }
    if (lane < M) dsc[lane] = si;
    __syncwarp();
    return true;
}

// H^-1 = D L^-T L^-1 D from hess_factor_regs's L^-1 (Lm) and D (dsc), by
// the whole block between two barriers (no warp waits on another's serial
// work here): entry (i, j) is s_i s_j times the dot product of columns i
// and j of L^-1.
template <int M, int NT>
__device__ __forceinline__ void hess_inverse_block(const double *Lm, const double *dsc, double *Hi) {
    for (int e = threadIdx.x; e < M * M; e += NT) {
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

}  // namespace
}  // namespace gpv
