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


@pytest.mark.parametrize("n", [255, 2048, 2049, 8192, 8193])
def test_one_launch_split_equals_host_partition(gpv_mod, n):
    """The device's split by segment: one block's share, the cluster's first
    round, one more, the largest batch of the single launch and the smallest
    of the counted one, given in a shuffled work order."""
    import torch
    from gpv import _lib, synth
    W = synth.workload(3, scale_down=4)
    rng = np.random.default_rng(n)
    pick = rng.integers(0, len(W["coords"]), n)
    d = gpv_mod.make_desc(W["coords"][pick], rng.choice([3, 5, 8, 21, 33, 49], n, p=[0.5, 0.2, 0.2, 0.06, 0.03, 0.01]),
                          rng.integers(0, 3, n), W["p0"][pick])
    d["p0"][d["order"] == 0, 2:] = 0.0
    d["radius"][5::97], d["order"][6::101] = 0, 3
    ctx = gpv_mod.Context(0)
    F, G = gpv_mod.Image(image_gs=W["f"], ctx=ctx), gpv_mod.Image(image_gs=W["g"], ctx=ctx)
    host = gpv_mod.solve_batch(F, G, d, max_iterations=4)
    ctx.reserve(n, int(d["radius"].max()), 4)
    dd = torch.from_numpy(d.view(np.uint8).copy()).cuda()
    order = torch.from_numpy(rng.permutation(n).astype(np.int32)).cuda()
    out = torch.zeros(n * _lib.RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    prm = gpv_mod._params(1e-5, 4, 0.75, False, gpv_mod.PREC_MIXED, None, None)
    for _ in range(2):  # the second finds the first's counts and queues
        out.zero_()
        _lib.check(_lib.lib().gpv_solve_batch_device(ctx.handle, F.handle, G.handle, ct.c_void_p(dd.data_ptr()),
                                                     ct.c_void_p(order.data_ptr()), n, ct.byref(prm),
                                                     ct.c_void_p(out.data_ptr()), None), "device batch")
        torch.cuda.synchronize()
        assert out.cpu().numpy().tobytes() == host.tobytes()
    assert np.all(host["status"][5::97] == 8) and np.all(host["status"][6::101] == 8)
