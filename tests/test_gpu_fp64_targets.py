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
