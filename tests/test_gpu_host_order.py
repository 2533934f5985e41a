"""A host batch brings its partition into launch segments with it; a device
batch makes it on the device.  Both return the same bytes, at the sizes where
the host's sort and the threads per subset change (one subset per SM, 4096
subsets), with subsets that no segment takes among them."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 148, 149, 5000])
def test_host_batches_equal_device_batches(gpv_mod, n):
    import torch
    from gpv import _lib, synth
    W = synth.workload(3, scale_down=4)
    rng = np.random.default_rng(n)
    pick = rng.integers(0, len(W["coords"]), n)
    d = gpv_mod.make_desc(W["coords"][pick], rng.integers(6, 34, n), rng.integers(0, 3, n), W["p0"][pick])
    d["p0"][d["order"] == 0, 2:] = 0.0
    if n > 2:
        d["radius"][1], d["order"][2] = 0, 7
    ctx = gpv_mod.Context(0)
    F, G = gpv_mod.Image(image_gs=W["f"], ctx=ctx), gpv_mod.Image(image_gs=W["g"], ctx=ctx)
    host = gpv_mod.solve_batch(F, G, d, max_iterations=12)
    ctx.reserve(n, int(d["radius"].max()), 12)
    dd = torch.from_numpy(d.view(np.uint8).copy()).cuda()
    out = torch.zeros(n * _lib.RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    prm = gpv_mod._params(1e-5, 12, 0.75, False, gpv_mod.PREC_MIXED, None, None)
    _lib.check(_lib.lib().gpv_solve_batch_device(ctx.handle, F.handle, G.handle, ct.c_void_p(dd.data_ptr()), None, n,
                                                 ct.byref(prm), ct.c_void_p(out.data_ptr()), None), "device batch")
    torch.cuda.synchronize()
    dev = out.cpu().numpy().view(_lib.RESULT_DTYPE)
    assert host.tobytes() == dev.tobytes()
    if n > 2:
        assert list(host["status"][1:3]) == [8, 8] and np.array_equal(host["p"][1], d["p0"][1])
