"""Singular and nearly singular Hessians of the FP64 solves
(csrc/icgn_runs64.cu): the Cholesky factor hands them to the elimination
with pivoting, which calls singular what has no pivot left, as the oracle does."""
import numpy as np
import pytest
from test_gpu_fp64_targets import BORDER, speckle

pytestmark = pytest.mark.gpu


def _case(gpv_mod, line):
    f = speckle()
    g = np.roll(f, (2, 1), (0, 1))
    i = np.arange(300)
    mask = np.zeros(f.shape, np.uint8)
    if line == "row":
        mask[150] = 1
        xy = [(c, 150) for c in range(60, 240)]
    elif line == "diagonal":
        mask[i, i] = 1
        xy = [(c, c) for c in range(60, 240)]
    else:  # two columns to a row
        mask[i[:150] * 2, i[:150]] = 1
        xy = [(c, 2 * c) for c in range(35, 115)]
    return f, g, mask, np.array(xy, float)


@pytest.mark.parametrize("line", ["row", "diagonal", "slope"])
@pytest.mark.parametrize("order", [1, 2])
def test_pixels_on_one_line_are_singular(oracle, gpv_mod, order, line):
    """With the template's pixels on one line the rows of dx and dy depend on
    each other.  On a row of the image dy is 0 and every pivot test sees it; on an
    oblique line the elimination reaches a zero pivot unless its own roundings
    differ (the oracle's never do here, this one's in one subset of thirty),
    where a factor that takes any positive residue for a pivot solved half of them."""
    f, g, mask, xy = _case(gpv_mod, line)
    p0 = np.zeros((len(xy), 12))
    p0[:, 0], p0[:, 1] = 1.1, 1.9
    d = gpv_mod.make_desc(xy, 20, order, p0)
    ref = oracle.solve_batch(oracle.get_c(f, BORDER), oracle.get_c(g, BORDER), f.shape, BORDER, d, mask=mask, max_iterations=1)
    assert np.all(ref["status"] == 3)
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
    M = gpv_mod.Mask("global", binary=mask)
    got = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, global_mask=M, max_iterations=1)
    assert np.array_equal(got["n_px"], ref["n_px"])
    assert (got["status"] == 3).mean() >= (1.0 if line == "row" else 0.9)
    if line == "row":
        fagn = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, global_mask=M, max_iterations=1, method="fagn")
        assert np.all(fagn["status"] == 3)


@pytest.mark.parametrize("order,method", [(0, "icgn"), (0, "fagn"), (1, "icgn"), (1, "fagn")])
def test_nearly_singular_matrices_are_solved(oracle, gpv_mod, order, method):
    """f = a(x + y) + 1e-6 b(x - y), moved by whole pixels: the scaled Hessian's
    last pivots are about 1e-12.  Order 0 finds the shift: along x + y as sharply as ever
    (1e-9 px); along x - y another prefilter's rounding, 1e-14 of 255, meets a
    signal of 1e-4 a pixel: 3e-8 px, so 1e-6 px.  (At order 1 the interpolation's
    own error is above that signal: only the copies are compared.)  Copies of
    a subset in one batch give the same bytes."""
    i = np.arange(300.0)
    X, Y = np.meshgrid(i, i)

    def image(u, v):
        s, t = X + Y - (u + v), X - Y - (u - v)
        return 120 + 40 * np.sin(s / 6.1) + 30 * np.sin(s / 9.7 + 1) + 1e-6 * (40 * np.sin(t / 2.9 + 2) + 30 * np.sin(t / 4.7))

    f, g = image(0, 0), image(1, -2)
    xy = np.repeat(np.array([[150.0, 150.0], [140.3, 160.6], [171.0, 133.7]]), 64, 0)
    p0 = np.zeros((len(xy), 12))
    p0[:, 0], p0[:, 1] = 1.05, -2.05
    d = gpv_mod.make_desc(xy, 25, order, p0)
    kw = dict(max_norm=1e-7, max_iterations=30, method=method)
    ref = oracle.solve_batch(oracle.get_c(f, BORDER), oracle.get_c(g, BORDER), f.shape, BORDER, d[::64], **kw)
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
    got = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, **kw)
    for k in range(3):
        same = got[64 * k:64 * k + 64]
        assert len(set(r.tobytes() for r in same)) == 1
    if order:
        return
    one = got[::64]
    assert np.all(ref["status"] == 0) and np.all(ref["converged"] == 1)
    assert np.array_equal(one["status"], ref["status"]) and np.array_equal(one["converged"], ref["converged"])
    for r in (ref, one):
        e = r["p"][:, :2] - [1.0, -2.0]
        assert np.abs(e.sum(1)).max() < 1e-9 and np.abs(e[:, 0] - e[:, 1]).max() < 1e-6


@pytest.mark.parametrize("order", [1, 2])
def test_fagn_elimination_is_read_after_it_is_written(gpv_mod, order):
    """FAGN's step by the elimination's inverse, which one lane writes and the
    others read: 128 copies of subsets that the factor rejects, the same bytes."""
    f, g, mask, xy = _case(gpv_mod, "slope")
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
    p0 = np.zeros((len(xy), 12))
    p0[:, 0], p0[:, 1] = 1.1, 1.9
    d = np.repeat(gpv_mod.make_desc(xy, 20, order, p0), 128)
    got = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, global_mask=gpv_mod.Mask("global", binary=mask),
                              max_iterations=1, method="fagn")
    for k in range(len(xy)):
        assert len(set(r.tobytes() for r in got[128 * k:128 * k + 128])) == 1, k


@pytest.mark.parametrize("method", ["icgn", "fagn"])
@pytest.mark.parametrize("order,share", [(1, 0.004), (1, 0.01), (2, 0.004), (2, 0.01)])
def test_subsets_of_fewer_pixels_than_parameters_converge_as_often(oracle, gpv_mod, order, share, method):
    """A sparse mask leaves a few pixels: the elimination inverts a rank-deficient
    matrix to its rounding, and the step is sound as long as the gradient is the
    direct sum over the residual.  Which subset converges turns on roundings; how many
    do, among 200 to 380, is the oracle's number within a fifth (two standard
    deviations of the smallest, 49)."""
    f = speckle(4)
    g = np.roll(f, (2, 1), (0, 1))
    r = np.random.default_rng(1)
    mask = (r.random(f.shape) < share).astype(np.uint8)
    xy = np.stack([r.integers(30, 270, 400), r.integers(30, 270, 400)], 1).astype(float)
    p0 = np.zeros((400, 12))
    p0[:, 0], p0[:, 1] = 1.1, 1.9
    d = gpv_mod.make_desc(xy, 12, order, p0)
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
    kw = dict(max_iterations=6, method=method)
    ref = oracle.solve_batch(F.coef(f64=True), G.coef(f64=True), f.shape, BORDER, d, mask=mask, **kw)
    got = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, global_mask=gpv_mod.Mask("global", binary=mask), **kw)
    few = (ref["n_px"] > 1) & (ref["n_px"] < {1: 6, 2: 12}[order])
    assert np.array_equal(got["n_px"], ref["n_px"]) and few.sum() >= 200
    assert got["converged"][few].sum() >= 0.8 * ref["converged"][few].sum()
