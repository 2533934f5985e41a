"""Workloads of the subset-correlation library, timed and compared.

Each case is one call (or one frame) as a program that uses the library makes
it: a single subset, a mesh, batches on the host and on the device, tracked
frames, image updates.  Inputs are seeded speckle pairs rendered on the GPU: a
blurred random field, displaced by a smooth field, with pixel noise.  The
workload sizes are those of this repository's benchmark and tests.

The fields of a mixed-precision solve (FP32 interpolation and residuals) are
returned in float32, those of the FP64 solves in float64; the iteration count
of a mixed solve, decided by the last bits of the norm it is compared with, is
left out, as is the norm itself.
"""
import ctypes as ct
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "geopyv-dev_b200"))

import gpv  # noqa: E402
from gpv import _lib  # noqa: E402
from gpv._lib import DESC_DTYPE, RESULT_DTYPE, SolveParams, check, lib  # noqa: E402

BORDER = 20
MAX_NORM, MAX_ITER, TOLERANCE = 1e-5, 50, 0.75
PARAMS = {0: 2, 1: 6, 2: 12}


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def batch(name, h, w, step, rmin, rmax, order, dtype="u8", field="quadratic", precision="mixed", method="icgn",
          texture="deformable", eta=False, call="device", grid="scattered"):
    """order 12: orders 1 and 2 mixed 70 / 30."""
    c = dict(kind="batch", h=h, w=w, step=step, rmin=rmin, rmax=rmax, order=order, dtype=dtype, field=field,
             precision=precision, method=method, texture=texture, eta=eta, call=call, grid=grid)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one subset picked by hand: the call a notebook makes, latency only
        dict(name="subset_r25", kind="subset", h=512, w=512, radius=25, order=1, dtype="u8", field="affine"),
        # a whole mesh solved by reliability-guided layers: a chain of small dependent batches
        dict(name="mesh_1600_layer_rg", kind="mesh", h=1024, w=1024, side=40, radius=25, order=1, dtype="u8",
             field="affine"),
        # first pass of a PIV run through the Python call: host descriptors in, host results out, with the diagnostic
        batch("host_o0_r16", 1024, 1024, 10, 16, 16, 0, field="shift", eta=True, call="host", grid="integer"),
        # the everyday strain map: first order, one megapixel, a grid every 20 px
        batch("batch_o1_r25", 1024, 1024, 20, 25, 25, 1, field="affine", grid="integer"),
        # the dense strain map of a 16-megapixel 12-bit pair: second order, a grid every 10 px
        batch("batch_o2_r30_16mp", 4096, 4096, 10, 30, 30, 2, dtype="u16"),
        # subsets of every size and both deformable orders, refined about a localised band
        batch("batch_band_r15_60", 2048, 2048, 9, 15, 60, 12, field="band"),
        # one frame of a tracked sequence: target prefiltered in place, 20k subsets seeded from the frame before
        dict(name="frame_20k_r25", kind="frame", h=2048, w=2048, step=14, radius=25, order=1, dtype="u8"),
        # the all-FP64 solve kept for calibration and verification runs
        batch("batch_fp64_o2_r30", 1024, 1024, 10, 30, 30, 2, dtype="u16", precision="fp64"),
        # forward additive Gauss-Newton, the package's second solver
        batch("batch_fagn_o1_r25", 1024, 1024, 20, 25, 25, 1, field="affine", method="fagn"),
        # speckle that moves rigidly with soil grains: the rigid-texture template
        batch("batch_rigid_o2_r30", 1531, 2047, 14, 30, 30, 2, texture="rigid"),
        # a new 16-megapixel frame: prefilter, then values and gradients at measuring points
        dict(name="image_u16_16mp", kind="image", h=4096, w=4096, dtype="u16", keep_f64=False, points=20000),
        # an odd-sized calibration image kept in FP64 and read in FP64
        dict(name="image_f64_odd", kind="image", h=911, w=1237, dtype="f64", keep_f64=True, points=5000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["mixed"] * 8 + ["fp64", "fagn", "rigid", "rigid", "host", "image", "image", "frame", "subset",
                                       "mesh"])
    dtype = rng.choice(["u8", "u16", "f32"])
    if what == "subset":
        order = rng.choice([0, 1, 2])
        return dict(kind="subset", h=_log(rng, 200, 1500), w=_log(rng, 200, 1500), radius=rng.randint(15 + 5 * order, 45),
                    order=order, dtype=dtype, field="shift" if order == 0 else "affine")
    if what == "image":
        keep = rng.random() < 0.4
        return dict(kind="image", h=_log(rng, 100, 4000), w=_log(rng, 100, 4000), keep_f64=keep,
                    dtype=rng.choice(["u8", "u16", "f32", "f64"]), points=_log(rng, 100, 20000))
    if what == "mesh":
        side = rng.randint(12, 45)
        return dict(kind="mesh", h=1024, w=1024 + rng.randint(0, 200), side=side, radius=rng.randint(18, 32),
                    order=rng.choice([1, 2]), dtype="u8", field="affine")
    if what == "frame":
        h, w = _log(rng, 500, 2048), _log(rng, 500, 2048)
        return dict(kind="frame", h=h, w=w, step=rng.randint(12, 24), radius=rng.randint(18, 32), order=1, dtype="u8")
    h, w = _log(rng, 256, 3000), _log(rng, 256, 3000)
    order = rng.choice([0, 1, 1, 2, 2, 12])
    if what == "rigid":
        order = rng.choice([1, 2])
    rmin = rng.randint({0: 10, 1: 14, 2: 22, 12: 22}[order], 40)
    rmin = min(rmin, (min(h, w) - 60) // 4)
    rmax = rmin if rng.random() < 0.6 else min(rmin + rng.randint(1, 25), (min(h, w) - 60) // 3)
    # subsets a case holds: by the work of the largest listed one, the FP64 forms at a twelfth of it
    most = 155000 * 2821 / (3.2 * rmax * rmax) / {"mixed": 1.3, "rigid": 3, "host": 4, "fp64": 15, "fagn": 25}[what]
    step = max(rng.randint(5, 24), math.ceil(math.sqrt(h * w / most)))
    return batch(None, h, w, step, rmin, rmax, order, dtype, field={0: "shift", 1: "affine", 2: "quadratic", 12: "band"}[order],
                 precision="fp64" if what == "fp64" else "mixed", method="fagn" if what == "fagn" else "icgn",
                 texture="rigid" if what == "rigid" else "deformable", eta=rng.random() < 0.25,
                 call="host" if what == "host" else "device", grid=rng.choice(["integer", "scattered"]))


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
SCALE = {"u8": 1.0, "u16": 16.0, "f32": 1.0, "f64": 1.0}
TORCH = {"u8": torch.uint8, "u16": torch.uint16, "f32": torch.float32, "f64": torch.float64}
CODE = {"u8": _lib.GPV_U8, "u16": _lib.GPV_U16, "f32": _lib.GPV_F32, "f64": _lib.GPV_F64}


def _gen(seed, k):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + k)


def _blur(a, sigma=1.7):
    n = math.ceil(4 * sigma)
    t = [math.exp(-0.5 * (i / sigma) ** 2) for i in range(-n, n + 1)]
    norm = math.sqrt(sum(v * v for v in t))
    for dim in (0, 1):
        size = a.shape[dim] - 2 * n
        a = sum(t[i] / norm * a.narrow(dim, i, size) for i in range(2 * n + 1))
    return a


def _speckle(h, w, seed):
    """Noise-free speckle, 30 to 200 grey levels, 24 px wider than the image on each side."""
    m = 24 + 7
    z = torch.randn(h + 2 * m, w + 2 * m, generator=_gen(seed, 1), device="cuda")
    return 30.0 + 170.0 * torch.sigmoid(2.0 * _blur(z))


def _field(case, seed, amount=1.0):
    """Displacement (u, v) and its gradient (ux, vx, uy, vy) at points, as functions of (x, y)."""
    r = np.random.default_rng(int(seed) + 77)
    t = r.uniform(-2, 2, 2)
    s = r.uniform(-1, 1, 6)
    xc, yc = case["w"] / 2.0, case["h"] / 2.0
    kind = case.get("field", "affine")
    a = np.zeros(4)  # ux, uy, vx, vy
    q = np.zeros(2)
    band = 0.0
    if kind != "shift":
        th = math.radians(0.5) * s[0]
        a = np.array([0.006 * s[1] + math.cos(th) - 1, -math.sin(th) + 0.003 * s[2], math.sin(th), 0.006 * s[3]])
    if kind == "quadratic":
        q = 1e-6 * np.array([1 + 0.3 * s[4], 1 + 0.3 * s[5]])
    if kind == "band":
        a, band = 0.3 * a, 1.5
    a, q, band, t = a * amount, q * amount, band * amount, t * amount

    def at(x, y):
        mod = torch if isinstance(x, torch.Tensor) else np
        dx, dy = x - xc, y - yc
        th = mod.tanh((y - yc) / 60.0)
        u = t[0] + a[0] * dx + a[1] * dy + q[0] * dx * dx + band * th
        v = t[1] + a[2] * dx + a[3] * dy + q[1] * dy * dy
        return u, v, (a[0] + 2 * q[0] * dx, a[2] + 0 * dx, a[1] + band / 60.0 * (1 - th * th), a[3] + 2 * q[1] * dy)
    return at


def _quantise(img, dtype, seed, k):
    img = SCALE[dtype] * (img + 2.0 * torch.randn(img.shape, generator=_gen(seed, k), device="cuda"))
    if dtype in ("u8", "u16"):
        top = 255.0 if dtype == "u8" else 4095.0
        return img.round().clamp(0.0, top).to(torch.int32).to(TORCH[dtype]).contiguous()
    return img.to(TORCH[dtype]).contiguous()


def _displaced(s, h, w, field):
    """The speckle seen after the displacement: g(X) = S(x) with x + u(x) = X."""
    X, Y = torch.meshgrid(torch.arange(w, device="cuda", dtype=torch.float64),
                          torch.arange(h, device="cuda", dtype=torch.float64), indexing="xy")
    x, y = X, Y
    for _ in range(4):
        u, v, _g = field(x, y)
        x, y = X - u, Y - v
    H, W = s.shape
    m = (H - h) // 2
    at = torch.stack([(x + m) * (2.0 / (W - 1)) - 1.0, (y + m) * (2.0 / (H - 1)) - 1.0], -1).float()
    return torch.nn.functional.grid_sample(s[None, None], at[None], mode="bicubic", padding_mode="border",
                                           align_corners=True)[0, 0]


def _pair(case, seed):
    h, w = case["h"], case["w"]
    s = _speckle(h, w, seed)
    field = _field(case, seed)
    m = (s.shape[0] - h) // 2
    f = _quantise(s[m:m + h, m:m + w], case["dtype"], seed, 2)
    return f, _quantise(_displaced(s, h, w, field), case["dtype"], seed, 3), field


def _desc(case, seed, field):
    """Centres on a grid, radii and orders of the case, first warps as a neighbour's solution gives them."""
    r = np.random.default_rng(int(seed) + 5)
    rmin, rmax = case.get("rmin", case.get("radius")), case.get("rmax", case.get("radius"))
    reach = 40 if case["field"] == "quadratic" and max(case["h"], case["w"]) > 2500 else 12
    m = min(rmax + 3 + reach, min(case["h"], case["w"]) // 2 - 1)
    X, Y = np.meshgrid(np.arange(m, case["w"] - m + 1e-9, case["step"]), np.arange(m, case["h"] - m + 1e-9, case["step"]))
    xy = np.stack([X.ravel(), Y.ravel()], 1).astype(np.float64)
    n = len(xy)
    if case.get("grid") != "integer":
        xy = xy + r.uniform(-0.5, 0.5, xy.shape)
    radius = np.exp(r.uniform(math.log(rmin), math.log(rmax + 0.49), n)).round().astype(np.int32).clip(rmin, rmax)
    order = np.full(n, case["order"], np.int32)
    if case["order"] == 12:
        order = np.where(r.uniform(size=n) < 0.7, 1, 2).astype(np.int32)
    u, v, g = field(xy[:, 0], xy[:, 1])
    p0 = np.zeros((n, 12))
    p0[:, 0], p0[:, 1] = u + r.uniform(-0.3, 0.3, n), v + r.uniform(-0.3, 0.3, n)
    for k in range(4):
        p0[:, 2 + k] = g[k]
    p0[order == 0, 2:] = 0.0
    return gpv.make_desc(xy, radius, order, p0)


def _image(ctx, px, keep_f64=False, grain=False, flip=False):
    px = px.cpu().numpy()
    return gpv.Image(image_gs=px[::-1] if flip else px, border=BORDER, ctx=ctx, keep_f64=keep_f64, grain=grain)


def _update(img, px, dtype):
    check(lib().gpv_image_update_device(img.handle, ct.c_void_p(px.data_ptr()), CODE[dtype]), "gpv_image_update_device")


class _Device:
    """Device memory of the library as a tensor."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3, strides=None)


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    s.kind = case["kind"]
    s.ctx = gpv.Context()
    s.stream = torch.cuda.ExternalStream(s.ctx.stream)
    if s.kind == "image":
        sp = _speckle(case["h"], case["w"], seed)
        m = (sp.shape[0] - case["h"]) // 2
        s.px = _quantise(sp[m:m + case["h"], m:m + case["w"]], case["dtype"], seed, 2)
        torch.cuda.synchronize()
        # the buffer's image holds an earlier frame
        s.img = _image(s.ctx, s.px, keep_f64=case["keep_f64"], flip=True)
        r = np.random.default_rng(int(seed))
        s.xy = r.uniform(0, 1, (case["points"], 2)) * [case["w"] - 1, case["h"] - 1]
        s.precision = gpv.PREC_FP64 if case["keep_f64"] else gpv.PREC_MIXED
        return s
    if s.kind == "frame":
        case = dict(case, field="affine", order=1)
        sp = _speckle(case["h"], case["w"], seed)
        m = (sp.shape[0] - case["h"]) // 2
        f = _quantise(sp[m:m + case["h"], m:m + case["w"]], case["dtype"], seed, 2)
        # the strain rises over four frames and falls again
        s.frames = [_quantise(_displaced(sp, case["h"], case["w"], _field(case, seed, a)), case["dtype"], seed, 3 + k)
                    for k, a in enumerate((0.25, 0.5, 0.75, 0.5))]
        s.f = _image(s.ctx, f)
        s.g = _image(s.ctx, f)
        s.desc = _desc(dict(case), seed, _field(case, seed, 0.25))
        s.seq = gpv.SubsetSequence(s.f, s.g, s.desc, np.uint8, max_norm=MAX_NORM, max_iterations=MAX_ITER)
        s.at = 0
        torch.cuda.synchronize()
        return s
    f, g, field = _pair(case, seed)
    if s.kind == "mesh":
        s.f, s.g = _image(s.ctx, f), _image(s.ctx, g)
        nodes, s.elements = _mesh(case)
        s.mesh = gpv.Mesh(nodes, s.elements, s.f, s.g)
        s.mask = gpv.Mask("local", shape="circle", size=case["radius"])
        k = len(nodes) // 2 + case["side"] // 2
        s.seed_at = [float(v) for v in nodes[k]]
        u, v, gr = field(nodes[k, 0], nodes[k, 1])
        s.seed_warp = [float(u), float(v)] + [float(q) for q in gr]
        return s
    if s.kind == "subset":
        s.f, s.g = _image(s.ctx, f), _image(s.ctx, g)
        d = _one(case, seed, field)
        s.subset = gpv.Subset(list(d["coord"][0]), gpv.Mask("local", shape="circle", size=case["radius"]), s.f, s.g,
                              subset_order=case["order"])
        s.p0 = d["p0"][0, :PARAMS[case["order"]]].copy()
        return s
    fp64 = case["precision"] == "fp64"
    rigid = case["texture"] == "rigid"
    s.f = _image(s.ctx, f, keep_f64=fp64, grain=rigid)
    s.g = _image(s.ctx, g, keep_f64=fp64)
    s.desc = _desc(case, seed, field)
    s.n = len(s.desc)
    if case["call"] == "device":
        flags = (_lib.SOLVE_ETA if case["eta"] else 0) | (_lib.SOLVE_FAGN if case["method"] == "fagn" else 0) | \
            (_lib.SOLVE_RIGID_TEXTURE if rigid else 0)
        s.params = SolveParams(max_norm=MAX_NORM, tolerance=TOLERANCE, max_iterations=MAX_ITER, flags=flags,
                               precision=gpv.PREC_FP64 if fp64 else gpv.PREC_MIXED, reserved=0, mask=None, history=None)
        s.ctx.reserve(s.n, case["rmax"], MAX_ITER)
        s.desc_dev = torch.from_numpy(s.desc.view(np.uint8).reshape(s.n, DESC_DTYPE.itemsize)).cuda()
        s.out = torch.zeros(s.n, RESULT_DTYPE.itemsize // 8, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return s


def _one(case, seed, field):
    at = np.array([[case["w"] * 0.47 + 0.31, case["h"] * 0.53 + 0.17]])
    u, v, g = field(at[:, 0], at[:, 1])
    p0 = np.zeros((1, 12))
    p0[0, :2] = u[0] + 0.2, v[0] - 0.15
    if case["order"]:
        p0[0, 2:6] = [float(np.ravel(q)[0]) for q in g]
    return gpv.make_desc(at, case["radius"], case["order"], p0)


def _mesh(case):
    """A structured mesh of side x side nodes, two triangles to a cell."""
    k, m = case["side"], case["radius"] + 30
    X, Y = np.meshgrid(np.linspace(m, case["w"] - m, k), np.linspace(m, case["h"] - m, k))
    i = np.arange(k * k).reshape(k, k)
    a, b, c, d = i[:-1, :-1].ravel(), i[:-1, 1:].ravel(), i[1:, :-1].ravel(), i[1:, 1:].ravel()
    return np.stack([X.ravel(), Y.ravel()], 1), np.concatenate([np.stack([a, b, c], 1), np.stack([b, d, c], 1)])


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def _from_device(out, f64, eta=False):
    """Fields of the results in device memory: n rows of 25 doubles, the last four of them eight 32-bit integers."""
    whole = out.view(torch.int32)
    if f64:
        r = {"warp_zncc": out[:, :14], "reference": out[:, 17:21], "counts": whole[:, 42:49]}
    else:
        r = {"warp_zncc": out[:, :13].float(), "reference": out[:, 17:21].float(), "counts": whole[:, 43:49]}
    if eta:
        r["eta"] = out[:, 15:17] if f64 else out[:, 15:17].float()
    return r


def run(s):
    case = s.case
    if s.kind == "batch" and case["call"] == "device":
        check(lib().gpv_solve_batch_device(s.ctx.handle, s.f.handle, s.g.handle, ct.c_void_p(s.desc_dev.data_ptr()), None,
                                           s.n, ct.byref(s.params), ct.c_void_p(s.out.data_ptr()),
                                           ct.c_void_p(s.ctx.stream)), "gpv_solve_batch_device")
        with torch.cuda.stream(s.stream):
            return _from_device(s.out, case["precision"] == "fp64" or case["method"] == "fagn", case["eta"])
    if s.kind == "batch":
        r = gpv.solve_batch(s.f, s.g, s.desc, max_norm=MAX_NORM, max_iterations=MAX_ITER, tolerance=TOLERANCE,
                            eta=case["eta"], precision=gpv.PREC_MIXED, method=case["method"], texture=case["texture"])
        return _from_host(r, case["eta"])
    if s.kind == "frame":
        s.seq.frame(device_ptr=s.frames[s.at % len(s.frames)].data_ptr(), download=False)
        s.at += 1
        out = torch.as_tensor(_Device(s.seq.results_device(), (s.seq.n, 25), "<f8"), device="cuda")
        with torch.cuda.stream(s.stream):
            # a copy: the memory is the tracker's own and holds the next frame's results soon
            return _from_device(out.clone(), False)
    if s.kind == "mesh":
        s.mesh.solve(s.mask, s.seed_at, s.seed_warp, max_norm=MAX_NORM, subset_order=case["order"],
                     preconditioning="layer-RG", layer_rg_max_workers=64)
        return _from_host(s.mesh.results, False)
    if s.kind == "subset":
        s.subset.solve(p_0=s.p0, max_norm=MAX_NORM)
        q = s.subset
        return {"warp": q.p.astype(np.float32), "zncc": np.float32(q.c_zncc), "eta": np.float32(q.eta_omitted),
                "reference": np.float32([q.f_m, q.delta_f, q.sssig, q.sigma_intensity]), "converged": int(q.converged)}
    _update(s.img, s.px, case["dtype"])
    val, grad = s.img.eval(s.xy, grad=True, precision=s.precision)
    if case["keep_f64"]:
        return {"value": val, "gradient": grad}
    return {"value": val.astype(np.float32), "gradient": grad.astype(np.float32)}


def _from_host(r, eta):
    got = {"warp": r["p"].astype(np.float32), "zncc": r["c_zncc"].astype(np.float32),
           "reference": np.stack([r[k] for k in ("f_m", "delta_f", "sssig", "sigma")], 1).astype(np.float32),
           "counts": np.stack([r[k] for k in ("converged", "quality_ok", "status", "n_px", "has_eta", "texture")], 1)}
    if eta:
        got["eta"] = np.stack([r["eta_u"], r["eta_v"]], 1).astype(np.float32)
    return got


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _disk(r):
    return int(sum(2 * math.isqrt(r * r - y * y) + 1 for y in range(-r, r + 1)))


def work(case):
    h, w = case["h"], case["w"]
    coef = (h + 2 * BORDER) * (w + 2 * BORDER)
    px = {"u8": 1, "u16": 2, "f32": 4, "f64": 8}[case["dtype"]] * h * w
    if case["kind"] == "image":
        # four first-order recursions per pass and pixel; 36 taps and their two derivatives per point
        return {"bytes": px + coef * (12 if case["keep_f64"] else 4) + case["points"] * 40,
                "flops": 2 * 8 * coef + 180 * case["points"]}
    # a target sample is 42 multiply-adds (36 taps, 6 row sums), with its gradient 90; a reference sample 90; five
    # iterations from a neighbour's warp, two more in a mesh's first ring, three from frame to frame
    each = 2 * 90 if case.get("method") == "fagn" else 2 * 42
    if case["kind"] == "subset":
        n, pixels, iters = 1, _disk(case["radius"]), 5
    elif case["kind"] == "mesh":
        n = case["side"] ** 2
        pixels, iters = n * _disk(case["radius"]), 5
    else:
        rmin, rmax = case.get("rmin", case.get("radius")), case.get("rmax", case.get("radius"))
        m = rmax + 15
        n = max(1, (h - 2 * m) // case["step"] + 1) * max(1, (w - 2 * m) // case["step"] + 1)
        rs = [int(round(math.exp(math.log(rmin) + (math.log(rmax + 0.49) - math.log(rmin)) * k / 63))) for k in range(64)]
        pixels, iters = n * sum(_disk(min(r, rmax)) for r in rs) / 64.0, 3 if case["kind"] == "frame" else 5
    size = 8 if case.get("precision") == "fp64" else 4
    extra = px + size * coef if case["kind"] == "frame" else 0
    return {"bytes": 2 * size * coef + n * (DESC_DTYPE.itemsize + RESULT_DTYPE.itemsize) + extra,
            "flops": pixels * (180 + each * iters)}


# --------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# --------------------------------------------------------------------------
Q = [[1 / 120, 13 / 60, 11 / 20, 13 / 60, 1 / 120, 0], [-1 / 24, -5 / 12, 0, 5 / 12, 1 / 24, 0],
     [1 / 12, 1 / 6, -1 / 2, 1 / 6, 1 / 12, 0], [-1 / 12, 1 / 6, 0, -1 / 6, 1 / 12, 0],
     [1 / 24, -1 / 6, 1 / 4, -1 / 6, 1 / 24, 0], [-1 / 120, 1 / 24, -1 / 12, 1 / 12, -1 / 24, 1 / 120]]


def _coefficients(px):
    """Quintic B-spline coefficients of the edge-padded image, by division of spectra."""
    a = torch.nn.functional.pad(px.to(torch.float64)[None, None], (BORDER,) * 4, mode="replicate")[0, 0]
    for dim in (0, 1):
        n = a.shape[dim]
        wj = 2.0 * math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n
        k = 11 / 20 + 13 / 30 * torch.cos(wj) + 1 / 60 * torch.cos(2 * wj)
        a = torch.fft.ifft(torch.fft.fft(a, dim=dim) / (k[:, None] if dim == 0 else k), dim=dim).real
    return a.contiguous()


def _weights(t, derivative):
    p = [torch.ones_like(t)]
    for _ in range(5):
        p.append(p[-1] * t)
    d = [0 * t] + [k * p[k - 1] for k in range(1, 6)]
    return [sum(Q[e][k] * (d if derivative else p)[e] for e in range(6) if Q[e][k]) for k in range(6)]


def _sample(c, h, w, x, y, grad):
    x, y = x.clamp(0.0, w - 1e-9), y.clamp(0.0, h - 1e-9)
    fx, fy = x.floor(), y.floor()
    at = (fy.long() + BORDER - 2) * c.shape[1] + fx.long() + BORDER - 2
    tx, ty = x - fx, y - fy
    a, b = _weights(ty, False), _weights(tx, False)
    if grad:
        da, db = _weights(ty, True), _weights(tx, True)
    flat = c.view(-1)
    v = gx = gy = 0.0
    for r in range(6):
        row = drow = 0.0
        for k in range(6):
            e = flat[at + (r * c.shape[1] + k)]
            row = row + b[k] * e
            if grad:
                drow = drow + db[k] * e
        v = v + a[r] * row
        if grad:
            gx, gy = gx + a[r] * drow, gy + da[r] * row
    return (v, gx, gy) if grad else v


def _shape(p, dx, dy, order):
    """Warped offsets of a batch of warps (b, 12) at template offsets."""
    c = [p[:, k, None] for k in range(12)]
    u, v = c[0] + 0 * dx, c[1] + 0 * dy
    if order >= 1:
        u, v = u + c[2] * dx + c[4] * dy, v + c[3] * dx + c[5] * dy
    if order == 2:
        u = u + 0.5 * c[6] * dx * dx + c[8] * dx * dy + 0.5 * c[10] * dy * dy
        v = v + 0.5 * c[7] * dx * dx + c[9] * dx * dy + 0.5 * c[11] * dy * dy
    return dx + u, dy + v


def _descent(gx, gy, dx, dy, order):
    mono = [torch.ones_like(gx)]
    if order >= 1:
        mono += [dx + 0 * gx, dy + 0 * gx]
    if order == 2:
        mono += [0.5 * dx * dx + 0 * gx, dx * dy + 0 * gx, 0.5 * dy * dy + 0 * gx]
    return torch.stack([q for m in mono for q in (gx * m, gy * m)], -1)


def _lift(q):
    u, v, ux, vx, uy, vy, uxx, vxx, uxy, vxy, uyy, vyy = (q[:, k] for k in range(12))
    z, o = torch.zeros_like(u), torch.ones_like(u)
    rows = [[1 + 2 * ux + ux * ux + u * uxx, 2 * u * uxy + 2 * (1 + ux) * uy, uy * uy + u * uyy, 2 * u * (1 + ux), 2 * u * uy,
             u * u],
            [0.5 * (v * uxx + 2 * (1 + ux) * vx + u * vxx), 1 + uy * vx + ux * vy + v * uxy + u * vxy + vy + ux,
             0.5 * (v * uyy + 2 * uy * (1 + vy) + u * vyy), v + v * ux + u * vx, u + v * uy + u * vy, u * v],
            [vx * vx + v * vxx, 2 * v * vxy + 2 * vx * (1 + vy), 1 + 2 * vy + vy * vy + v * vyy, 2 * v * vx,
             2 * v * (1 + vy), v * v],
            [0.5 * uxx, uxy, 0.5 * uyy, 1 + ux, uy, u], [0.5 * vxx, vxy, 0.5 * vyy, vx, 1 + vy, v], [z, z, z, z, z, o]]
    return torch.stack([torch.stack(r, -1) for r in rows], -2)


def _compose(p, dp, order):
    """The warp after the inverse of the increment."""
    out = torch.zeros_like(p)
    if order == 0:
        out[:, :2] = p[:, :2] - dp[:, :2]
        return out
    n = (_lift(p) @ torch.linalg.inv(_lift(dp)))
    for k, (i, j, f, s) in enumerate([(3, 5, 1, 0), (4, 5, 1, 0), (3, 3, 1, 1), (4, 3, 1, 0), (3, 4, 1, 0), (4, 4, 1, 1),
                                      (3, 0, 2, 0), (4, 0, 2, 0), (3, 1, 1, 0), (4, 1, 1, 0), (3, 2, 2, 0), (4, 2, 2, 0)]):
        if k < PARAMS[order]:
            out[:, k] = f * n[:, i, j] - s
    return out


def _grain(px):
    """Second derivatives of the smoothed image over its speckle size, and that size's square."""
    a = px.to(torch.float64)
    h, w = a.shape
    side = min(512, h, w) & ~1
    r0, c0 = h // 2 - side // 2, w // 2 - side // 2
    crop = a[r0:r0 + side, c0:c0 + side]
    crop = crop - crop.mean()
    ac = torch.fft.ifft2(torch.fft.fft2(crop).abs() ** 2).real
    prof = (0.5 * (ac[0, :side // 2] + ac[:side // 2, 0]) / ac[0, 0]).cpu().numpy()
    k = int(np.argmax(prof < 0.5))
    ell = k - 1 + (prof[k - 1] - 0.5) / (prof[k - 1] - prof[k])
    s2 = ell * ell / (2 * math.log(2.0))
    i = torch.arange(-4, 5, device="cuda", dtype=torch.float64)
    g = torch.exp(-i * i / 2) / torch.exp(-i * i / 2).sum()
    taps = [g, i * g, (i * i - 1) * g]

    def along(b, t, dim):
        b = torch.nn.functional.pad(b[None, None], (4, 4, 0, 0) if dim else (0, 0, 4, 4), mode="replicate")[0, 0]
        return sum(t[j] * b.narrow(dim, j, a.shape[dim]) for j in range(9))
    corr = ((s2 / 2 + 1) / (s2 / 2)) ** 2
    return s2, [corr * along(along(a, taps[x], 1), taps[y], 0) for x, y in ((2, 0), (0, 2), (1, 1))]


def _bilinear(m, x, y):
    h, w = m.shape
    x, y = x.clamp(0.0, w - 1.0), y.clamp(0.0, h - 1.0)
    x0, y0 = x.floor().clamp(max=w - 2).long(), y.floor().clamp(max=h - 2).long()
    tx, ty = x - x0, y - y0
    q = m.reshape(-1)
    at = y0 * w + x0
    return (1 - ty) * ((1 - tx) * q[at] + tx * q[at + 1]) + ty * ((1 - tx) * q[at + w] + tx * q[at + w + 1])


def _solve(f, g, desc, method="icgn", texture="deformable", max_norm=MAX_NORM):
    """Warps (n, 12), ZNCC (n), ZNSSD (n) and (mean, spread, gradient sum, deviation) (n, 4) in 64 bits."""
    h, w = f.shape
    cf, cg = _coefficients(f), _coefficients(g)
    grain = _grain(f) if texture == "rigid" else None
    n = len(desc)
    warp = torch.zeros(n, 12, dtype=torch.float64, device="cuda")
    zn = torch.zeros(n, 2, dtype=torch.float64, device="cuda")
    ref = torch.zeros(n, 4, dtype=torch.float64, device="cuda")
    keys = desc["order"].astype(np.int64) * 100000 + desc["radius"]
    for key in np.unique(keys):
        order, r = int(key // 100000), int(key % 100000)
        M = PARAMS[order]
        yy, xx = np.mgrid[-r:r + 1, -r:r + 1]
        keep = xx * xx + yy * yy <= r * r
        dx = torch.from_numpy(xx[keep].astype(np.float64)).cuda()[None]
        dy = torch.from_numpy(yy[keep].astype(np.float64)).cuda()[None]
        px = dx.shape[1]
        which = np.nonzero(keys == key)[0]
        for lo in range(0, len(which), max(1, 5_000_000 // px)):
            at = which[lo:lo + max(1, 5_000_000 // px)]
            d = desc[at]
            c = torch.from_numpy(d["coord"].copy()).cuda()
            cx, cy = c[:, :1], c[:, 1:]
            p = torch.from_numpy(d["p0"].copy()).cuda()
            p[:, M:] = 0.0
            v, gx, gy = _sample(cf, h, w, cx + dx, cy + dy, True)
            fm = v.mean(1, keepdim=True)
            a0 = v - fm
            df = a0.square().sum(1, keepdim=True).sqrt()
            sd = _descent(gx, gy, dx, dy, order)
            hinv = torch.linalg.inv(sd.transpose(1, 2) @ sd)
            sums = torch.stack([fm[:, 0], df[:, 0], 0.5 * (gx * gx + gy * gy).sum(1), df[:, 0] / math.sqrt(px)], 1)
            if grain:
                hs = [_bilinear(m, cx + dx, cy + dy) for m in grain[1]]
            live = torch.ones(len(at), dtype=torch.bool, device="cuda")
            z = torch.zeros(len(at), dtype=torch.float64, device="cuda")
            for _ in range(MAX_ITER):
                ox, oy = _shape(p, dx, dy, order)
                if method == "fagn":
                    gv, hx, hy = _sample(cg, h, w, cx + ox, cy + oy, True)
                else:
                    gv = _sample(cg, h, w, cx + ox, cy + oy, False)
                a, dt = a0, df
                if grain:
                    q = [p[:, k, None] for k in range(12)]
                    ux, vx = q[2] + q[6] * dx + q[8] * dy, q[3] + q[7] * dx + q[9] * dy
                    uy, vy = q[4] + q[8] * dx + q[10] * dy, q[5] + q[9] * dx + q[11] * dy
                    e0, e1 = ux + 0.5 * (ux * ux + vx * vx), vy + 0.5 * (uy * uy + vy * vy)
                    e2 = 0.5 * (uy + vx) + 0.5 * (ux * uy + vx * vy)
                    t = v - 0.5 * grain[0] * (e0 * hs[0] + e1 * hs[1] + 2 * e2 * hs[2]) - (e0 + e1) * a0
                    a = t - t.mean(1, keepdim=True)
                    dt = a.square().sum(1, keepdim=True).sqrt()
                b = gv - gv.mean(1, keepdim=True)
                dg = b.square().sum(1, keepdim=True).sqrt()
                zs = (a / dt - b / dg).square().sum(1)
                if method == "fagn":
                    sg = _descent(hx, hy, ox - p[:, :1], oy - p[:, 1:2], order)
                    dp = torch.linalg.solve(sg.transpose(1, 2) @ sg, (sg * (a * dg / dt - b)[..., None]).sum(1))
                else:
                    dp = -(hinv @ (sd * (a - dt / dg * b)[..., None]).sum(1)[..., None])[..., 0]
                full = torch.nn.functional.pad(dp, (0, 12 - M))
                new = p + full if method == "fagn" else _compose(p, full, order)
                scale = torch.tensor([1.0] * 2 + [math.sqrt(px)] * 4 + [0.5 * px] * 6, dtype=torch.float64, device="cuda")
                norm = (full * scale).square().sum(1).sqrt()
                p = torch.where(live[:, None], new, p)
                z = torch.where(live, zs, z)
                live = live & ~(norm < max_norm)
                if not bool(live.any()):
                    break
            i = torch.from_numpy(at).cuda()
            warp[i], ref[i] = p, sums
            zn[i, 0], zn[i, 1] = 1 - z / 2, z
    return warp, zn[:, 0], zn[:, 1], ref


def exact(case, seed):
    if case["kind"] == "image":
        sp = _speckle(case["h"], case["w"], seed)
        m = (sp.shape[0] - case["h"]) // 2
        px = _quantise(sp[m:m + case["h"], m:m + case["w"]], case["dtype"], seed, 2)
        r = np.random.default_rng(int(seed))
        xy = torch.from_numpy(r.uniform(0, 1, (case["points"], 2)) * [case["w"] - 1, case["h"] - 1]).cuda()
        v, gx, gy = _sample(_coefficients(px), case["h"], case["w"], xy[:, 0], xy[:, 1], True)
        return {"value": v, "gradient": torch.stack([gx, gy], 1)}
    if case["kind"] == "frame":
        full = dict(case, field="affine", order=1)
        sp = _speckle(case["h"], case["w"], seed)
        m = (sp.shape[0] - case["h"]) // 2
        f = _quantise(sp[m:m + case["h"], m:m + case["w"]], case["dtype"], seed, 2)
        field = _field(full, seed, 0.25)
        g = _quantise(_displaced(sp, case["h"], case["w"], field), case["dtype"], seed, 3)
        warp, zncc, _, ref = _solve(f, g, _desc(full, seed, field))
        return {"warp_zncc": torch.cat([warp, zncc[:, None]], 1), "reference": ref, "counts": None}
    f, g, field = _pair(case, seed)
    if case["kind"] == "mesh":
        # the fixed point that the nodes' solves end at, whatever neighbour they started from
        nodes, _ = _mesh(case)
        u, v, gr = field(nodes[:, 0], nodes[:, 1])
        p0 = np.stack([u, v, *gr], 1)
        warp, zncc, _, ref = _solve(f, g, gpv.make_desc(nodes, case["radius"], case["order"], p0), max_norm=1e-8)
        return {"warp": warp, "zncc": zncc, "reference": ref, "counts": None}
    if case["kind"] == "subset":
        warp, zncc, _, ref = _solve(f, g, _one(case, seed, field))
        return {"warp": warp[0, :PARAMS[case["order"]]], "zncc": zncc[0], "reference": ref[0], "eta": None,
                "converged": None}
    warp, zncc, znssd, ref = _solve(f, g, _desc(case, seed, field), case["method"], case["texture"])
    if case["call"] == "host":
        return {"warp": warp, "zncc": zncc, "reference": ref, "counts": None, "eta": None}
    both = [warp, zncc[:, None]]
    if case["precision"] == "fp64" or case["method"] == "fagn":
        both.append(znssd[:, None])
    got = {"warp_zncc": torch.cat(both, 1), "reference": ref, "counts": None}
    return dict(got, eta=None) if case["eta"] else got
