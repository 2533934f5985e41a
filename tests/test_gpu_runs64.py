"""The FP64 run-layout solves (csrc/icgn_runs64.cu) against the oracle where
their layout has edges: radii around a band's four rows, the switch to 256
threads above radius 32, windows that do not fit in shared memory (radius 90),
subsets at the image's edge, and FP32 coefficients widened at staging (FAGN).

Tolerances are those of the FP64 forms elsewhere: 1e-9 px, 1e-11 in the
gradients, 1e-10 in ZNCC for ICGN (test_gpu_icgn), 1e-8 for FAGN on FP64
coefficients and 1e-3 px on FP32 ones (test_gpu_fagn)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BORDER = 20


def _case(gpv_mod, oracle, keep=True):
    from gpv import synth
    W = synth.workload(2, scale_down=16)
    F = gpv_mod.Image(image_gs=W["f"], border=BORDER, keep_f64=keep)
    G = gpv_mod.Image(image_gs=W["g"], border=BORDER, keep_f64=keep)
    return W, F, G, oracle.get_c(W["f"].astype(np.float64), BORDER), oracle.get_c(W["g"].astype(np.float64), BORDER)


def _desc(gpv_mod, W, radius, order):
    from gpv import synth
    n = W["f"].shape[0]
    # inside (when the radius allows it), and overhanging two edges
    xy = np.array([[n / 2 + 0.31, n / 2 - 0.43], [n / 2 - 7.0, n / 2 + 5.0], [radius * 0.8, n / 2 + 1.3],
                   [n / 2 - 3.7, n - 1 - radius * 0.7]])
    p0 = synth.seeded_p0(W["field"], xy, np.random.default_rng(radius), 0.2)
    p0[:, {0: 2, 1: 6, 2: 12}[order]:] = 0.0
    return gpv_mod.make_desc(xy, radius, order, p0)


@pytest.mark.parametrize("radius,order", [(1, 0), (2, 0), (3, 0), (4, 0), (12, 1), (13, 1), (32, 2), (33, 2), (34, 1),
                                          (77, 1), (90, 2)])
def test_icgn_fp64(gpv_mod, oracle, radius, order):
    W, F, G, Cf, Cg = _case(gpv_mod, oracle)
    d = _desc(gpv_mod, W, radius, order)
    kw = dict(max_norm=1e-5, max_iterations=25, eta=True)
    ref = oracle.solve_batch(Cf, Cg, W["f"].shape, BORDER, d, **kw)
    got = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, **kw)
    for k in ("status", "n_px", "converged", "quality_ok"):
        assert np.array_equal(got[k], ref[k]), k
    ok = (ref["status"] == 0) & (ref["converged"] == 1)
    assert ok.any() or radius <= 3  # the oracle itself does not settle on some of the smallest subsets
    assert np.array_equal(got["iterations"][ok], ref["iterations"][ok])
    dp = np.abs(got["p"] - ref["p"])[ok]
    if ok.any():
        assert dp[:, :2].max() < 1e-9 and dp[:, 2:].max() < 1e-11
        assert np.abs(got["c_zncc"] - ref["c_zncc"])[ok].max() < 1e-10
        assert np.abs(got["c_znssd"] - ref["c_znssd"])[ok].max() < 2e-10
        assert np.abs(got["eta_u"] - ref["eta_u"])[ok].max() < 1e-9


@pytest.mark.parametrize("keep", [True, False], ids=["f64", "f32"])
@pytest.mark.parametrize("radius,order", [(4, 0), (13, 1), (32, 2), (34, 2), (90, 1)])
def test_fagn(gpv_mod, oracle, radius, order, keep):
    W, F, G, Cf, Cg = _case(gpv_mod, oracle, keep)
    d = _desc(gpv_mod, W, radius, order)
    kw = dict(max_norm=1e-5, max_iterations=25, eta=True, method="fagn")
    ref = oracle.solve_batch(Cf, Cg, W["f"].shape, BORDER, d, **kw)
    got = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64 if keep else gpv_mod.PREC_MIXED, **kw)
    ok = (ref["status"] == 0) & (ref["converged"] == 1) & (got["iterations"] == ref["iterations"])
    assert np.array_equal(got["status"], ref["status"]) and np.array_equal(got["converged"], ref["converged"])
    assert ok.any()
    dp = np.abs(got["p"] - ref["p"])[ok]
    if keep:
        assert dp.max() < 1e-8 and np.abs(got["eta_u"] - ref["eta_u"])[ok].max() < 1e-8
    else:
        assert dp[:, :2].max() <= 1e-3 and dp[:, 2:6].max() <= 1e-5


def test_singular_matrices_are_judged_by_the_pivoted_elimination(gpv_mod, oracle):
    """Fewer pixels than parameters: the factor has no positive pivot left; what the pivoted elimination
    accepts is still solved, so only the status of a matrix without a pivot says singular."""
    W, F, G, Cf, Cg = _case(gpv_mod, oracle)
    n = W["f"].shape[0]
    d = gpv_mod.make_desc([[n / 2 + 0.3, n / 2 + 0.4], [n / 2 - 20.0, n / 2 + 9.0]], 1, 1)
    got = gpv_mod.solve_batch(F, G, d, precision=gpv_mod.PREC_FP64, max_iterations=3)
    assert set(got["status"]) <= {0, 3, 4, 5} and np.all(got["n_px"] == 5)
