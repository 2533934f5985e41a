"""FP64 solves (csrc/icgn_runs64.cu) on targets without contrast, or with a grey
level far from the reference's: areas of zero, saturated areas, and what a
warp past a corner of the image reads, which is one clamped value.

A target without contrast correlates with nothing: the ZNCC is undefined (NaN)
where the target is constant to the last bit, and the correlation of n
samples with rounding noise, about n^-1/2, where it is not.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BORDER = 20


def speckle(seed=99, n=300):
    r = np.random.default_rng(seed)
    a = r.standard_normal((n + 40, n + 40))
    k = np.exp(-0.5 * (np.arange(-7, 8) / 1.7) ** 2)
    k /= np.sqrt((k * k).sum())
    for ax in (0, 1):
        a = np.apply_along_axis(lambda v: np.convolve(v, k, "same"), ax, a)
    return 120.0 + 40.0 * a[20:-20, 20:-20]


def desc(gpv_mod, shifts, order, radius=20, at=(120.3, 140.6)):
    p0 = np.zeros((len(shifts), 12))
    p0[:, :2] = shifts
    return gpv_mod.make_desc(np.tile([at], (len(shifts), 1)), radius, order, p0)


@pytest.mark.parametrize("order", [0, 1, 2])
def test_zero_target_gives_no_correlation(gpv_mod, order):
    """A target that is exactly zero under the subset (more than the
    prefilter's reach from its edge): delta_g is 0 and the ZNSSD undefined."""
    f = speckle()
    g = f.copy()
    g[:, 100:] = 0.0
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
    d = desc(gpv_mod, [(100.0, 0.0), (110.3, 5.2), (120.0, -7.5)], order)
    for its in (1, 5):
        got, hist = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, max_iterations=its, history=True)
        assert not got["converged"].any() and not got["quality_ok"].any()
        # order 0 steps by NaN and ends not finite; the others cannot compose that step and keep the first warp
        assert np.all(got["status"] == (5 if order == 0 else 4))
        if order == 0:
            assert np.isnan(got["c_zncc"]).all() and np.isnan(got["c_znssd"]).all()
            assert np.isnan(hist[:, 0, 1:]).all()
        else:
            assert np.all(got["c_zncc"] == 0.0) and np.all(got["c_znssd"] == 4.0)


@pytest.mark.parametrize("method", ["icgn", "fagn"])
@pytest.mark.parametrize("order", [0, 1, 2])
def test_target_without_contrast_is_never_a_match(gpv_mod, order, method):
    """Saturated areas and warps past each corner (every sample reads the
    corner's value): the target's spread is its own rounding, not what two
    large sums about f's mean leave of each other."""
    f = speckle()
    sat = f.copy()
    sat[:, 150:] = 255.0
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    for g, shifts in ((sat, [(100.0, 0.0), (110.3, 5.2), (120.0, -7.5)]),
                      (f, [(-400.0, -400.0), (400.0, -400.0), (-400.0, 400.0), (400.0, 400.0)])):
        G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
        d = desc(gpv_mod, shifts, order)
        for its in (1, 5) if method == "icgn" else (1,):  # (FAGN's second warp may be anywhere)
            got, hist = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, method=method, max_iterations=its,
                                            history=True)
            assert not got["quality_ok"].any()
            # correlations with rounding noise are of the size n^-1/2 = 0.03
            for z in (got["c_zncc"], hist[:, :, 1]):
                assert np.all(np.isnan(z) | (np.abs(z) < 0.5)), (z, got["status"])


@pytest.mark.parametrize("order", [0, 1, 2])
def test_zero_target_ends_at_the_first_iteration(gpv_mod, order):
    """On zeros the spread is exactly 0 whatever f's mean: the step is NaN."""
    f = speckle()
    g = f.copy()
    g[:, 100:] = 0.0
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
    got, hist = gpv_mod.solve_batch(F, G, desc(gpv_mod, [(100.0, 0.0), (110.3, 5.2), (120.0, -7.5)], order),
                                    precision=gpv_mod.PREC_FP64, max_iterations=5, history=True)
    assert np.all(got["status"] == (5 if order == 0 else 4)) and np.all(got["iterations"] == (1 if order == 0 else 0))
    assert np.isnan(hist[:, 0]).all() == (order == 0) and np.all(hist[:, 1:] == 0.0)


@pytest.mark.parametrize("method", ["icgn", "fagn"])
@pytest.mark.parametrize("order", [0, 1, 2])
def test_target_of_another_level_costs_no_digits(oracle, gpv_mod, order, method):
    """A target 1e5 of its contrasts away from f_m, one iteration (the level of
    the next ones is the target's own): 1e-9 px and 1e-10 in ZNCC as elsewhere;
    one sum about f_m leaves 1e-6 and 1e-6."""
    a = (speckle() - 120.0) / 40.0
    f, g = a + 5.0, np.roll(a, (2, 1), (0, 1)) + 1e5
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
    p0 = np.zeros((3, 12))
    p0[:, 0], p0[:, 1] = 1.1, 1.9
    d = gpv_mod.make_desc([[120.3, 140.6], [150.0, 150.0], [170.2, 133.3]], 20, order, p0)
    kw = dict(max_iterations=1, history=True, method=method)
    ref, rh = oracle.solve_batch(oracle.get_c(f, BORDER), oracle.get_c(g, BORDER), f.shape, BORDER, d, **kw)
    got, gh = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, **kw)
    assert np.array_equal(got["status"], ref["status"])
    assert np.abs(got["p"][:, :2] - ref["p"][:, :2]).max() < 1e-9
    assert np.abs(got["c_zncc"] - ref["c_zncc"]).max() < 1e-10
    assert np.abs(gh[:, 0, 1:] - rh[:, 0, 1:]).max() < 2e-10


@pytest.mark.parametrize("method", ["icgn", "fagn"])
@pytest.mark.parametrize("order", [0, 1, 2])
def test_warps_past_the_range_of_an_int_read_the_same_edge(gpv_mod, order, method):
    """Every sample of a warp past an edge reads that edge, however far it is
    (src/image.rs:129-132): 3e9 px and an infinity give the sums of 4e4 px."""
    f = speckle()
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=np.roll(f, (2, 1), (0, 1)), border=BORDER, keep_f64=True)
    way = np.array([(1, 0), (-1, 0), (0, 1), (0, -1)], float)
    res = []
    for far in (4e4, 3e9, np.inf):
        shifts = np.where(way == 0.0, 0.25, np.copysign(far, way))
        res.append(gpv_mod.solve_batch(F, G, desc(gpv_mod, shifts, order), precision=gpv_mod.PREC_FP64, method=method,
                                       max_iterations=1))
        assert np.all(res[-1]["c_zncc"] != 0.0)  # a row or a column of the image is not without contrast
    for r in res[1:]:
        for k in ("c_zncc", "c_znssd", "status", "iterations"):
            assert np.array_equal(r[k], res[0][k]), k


@pytest.mark.parametrize("order", [1, 2])
def test_strains_past_the_range_of_an_int_read_both_edges(gpv_mod, order):
    f = speckle()
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=np.roll(f, (2, 1), (0, 1)), border=BORDER, keep_f64=True)
    res = []
    for ux in (1e5, 1e9, 1e12):
        d = desc(gpv_mod, [(0.3, 0.2), (0.3, 0.2)], order)
        d["p0"][0, 2], d["p0"][1, 5] = ux, -ux
        res.append(gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, max_iterations=1))
        assert np.all(res[-1]["c_zncc"] != 0.0)
    for r in res[1:]:
        assert np.array_equal(r["c_zncc"], res[0]["c_zncc"]) and np.array_equal(r["status"], res[0]["status"])


@pytest.mark.parametrize("method", ["icgn", "fagn"])
@pytest.mark.parametrize("order", [0, 1, 2])
def test_masked_hot_centre_costs_no_digits(oracle, gpv_mod, order, method):
    """A pixel of 1e8 in f that the mask leaves out with 24 px around it: f_m,
    delta_f and the solve are those of the remaining pixels, 1e-9 px and 1e-10
    in ZNCC of the oracle's as elsewhere, from the same coefficients (another
    prefilter's rounding of such a pixel is 1e-8 near it)."""
    f = speckle()
    g = np.roll(f, (2, 1), (0, 1))
    f[140, 120] = 1e8
    mask = np.ones(f.shape, np.uint8)
    mask[116:165, 96:145] = 0
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=True)
    d = desc(gpv_mod, [(1.1, 1.9)], order, radius=45, at=(120.0, 140.0))
    kw = dict(max_iterations=3, history=True, method=method)
    got, gh = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, global_mask=gpv_mod.Mask("global", binary=mask), **kw)
    ref, rh = oracle.solve_batch(F.coef(f64=True), G.coef(f64=True), f.shape, BORDER, d, mask=mask, **kw)
    assert got["n_px"][0] == ref["n_px"][0] > 3000 and np.array_equal(got["status"], ref["status"])
    assert abs(got["delta_f"][0] / ref["delta_f"][0] - 1) < 1e-12 and abs(got["f_m"][0] - ref["f_m"][0]) < 1e-10
    assert np.abs(got["p"][:, :2] - ref["p"][:, :2]).max() < 1e-9
    assert np.abs(got["c_zncc"] - ref["c_zncc"]).max() < 1e-10
    assert np.abs(gh[0, :, 1:] - rh[0, :, 1:]).max() < 2e-10


@pytest.mark.parametrize("keep", [True, False], ids=["f64", "f32"])
@pytest.mark.parametrize("area", ["whole", "half"])
def test_fagn_on_a_saturated_target_is_not_singular(oracle, gpv_mod, area, keep):
    """A translation over equal coefficients: the target's gradient is its rounding,
    not exactly 0, so no subset is called singular (which would end a mesh)."""
    f = speckle()
    g = np.full(f.shape, 255.0)
    if area == "half":
        g[:, :100] = f[:, :100]
    r = np.random.default_rng(5)
    xy = np.stack([r.uniform(190, 260, 200), r.uniform(40, 260, 200)], 1)
    p0 = np.zeros((200, 12))
    p0[:, :2] = r.uniform(-3, 3, (200, 2))
    d = gpv_mod.make_desc(xy, 15, 0, p0)
    kw = dict(method="fagn", max_iterations=1)
    ref = oracle.solve_batch(oracle.get_c(f, BORDER), oracle.get_c(g, BORDER), f.shape, BORDER, d, **kw)
    assert np.all(ref["status"] == 0)
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=keep)
    G = gpv_mod.Image(image_gs=g, border=BORDER, keep_f64=keep)
    got = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64 if keep else gpv_mod.PREC_MIXED, **kw)
    assert (got["status"] == 0).mean() >= 0.95  # (a sum of roundings may still be 0: one in 200 with the kernel before the run layout)


@pytest.mark.parametrize("method", ["icgn", "fagn"])
def test_reference_statistics_next_to_a_pixel_that_is_nan(gpv_mod, method):
    """A NaN pixel in f reaches 44 samples: subsets inside that square and across
    its edge are featureless with f_m NaN, delta_f 0 where no pixel is a number
    and NaN where some are; 45 samples away they are as without it."""
    f = speckle()
    clean = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    f = f.copy()
    f[150, 150] = np.nan
    F = gpv_mod.Image(image_gs=f, border=BORDER, keep_f64=True)
    G = gpv_mod.Image(image_gs=np.roll(speckle(), (2, 1), (0, 1)), border=BORDER, keep_f64=True)
    # a sample reads coefficients from 2 before to 3 after it
    d = gpv_mod.make_desc([[150, 150], [150 + 44, 150], [150, 150 - 45 - 13], [150 + 45 + 12, 150]], 10, 1,
                          [[1.1, 1.9] + [0.0] * 10] * 4)
    kw = dict(precision=gpv_mod.PREC_FP64, method=method)
    got, ref = gpv_mod.solve_batch(F, G, d, **kw), gpv_mod.solve_batch(clean, G, d, **kw)
    assert list(got["status"]) == [2, 2, 0, 0] and np.all(np.isnan(got["f_m"][:2]))
    assert got["delta_f"][0] == 0.0 and np.isnan(got["delta_f"][1])
    assert np.abs(got["p"][2:] - ref["p"][2:]).max() < 1e-9 and np.abs(got["delta_f"][2:] / ref["delta_f"][2:] - 1).max() < 1e-12


@pytest.mark.parametrize("order", [1, 2])
def test_a_mesh_over_a_saturated_half_is_solved(gpv_mod, order):
    """FAGN on FP32 coefficients: nodes on the saturated half are not called
    singular, which would end the mesh, nor matched; the others are solved."""
    f = speckle(3, 400).round().clip(0, 255)
    g = np.roll(f, (1, 2), (0, 1))
    g[:, 230:] = 255.0
    X, Y = np.meshgrid(np.linspace(50, 350, 9), np.linspace(50, 350, 9))
    nodes = np.stack([X.ravel(), Y.ravel()], 1)
    i = np.arange(81).reshape(9, 9)
    a, b, c, e = i[:-1, :-1].ravel(), i[:-1, 1:].ravel(), i[1:, :-1].ravel(), i[1:, 1:].ravel()
    elements = np.concatenate([np.stack([a, b, c], 1), np.stack([b, e, c], 1)])
    m = gpv_mod.Mesh(nodes, elements, gpv_mod.Image(image_gs=f), gpv_mod.Image(image_gs=g))
    m.solve(20, [87.5, 87.5], [2.0, 1.0] + [0.0] * (6 * order - 2), subset_order=order, method="fagn",
            preconditioning="layer-RG", override_active=True)
    assert m.quality_ok[nodes[:, 0] < 200].all() and not m.quality_ok[nodes[:, 0] > 260].any()
    assert np.all(m.c_zncc[nodes[:, 0] > 260] < 0.75)
