"""What is timed, and against what it is checked: reconstructions as a user of
sscRaft runs them, through its public entry points.

Each case is one call (or, for the network, one training step).  Device cases
pass torch CUDA tensors to the library's device entries, as a program that keeps
its scan on the GPU does; the host case passes numpy arrays to `sscRaft.fbp`.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as tf

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ssc-raft_b200"))

import sscRaft  # noqa: E402
from sscRaft.rafttypes import FilterNumber, check_error, libraft  # noqa: E402
from sscRaft.warmstart import UNet, default_weights, input_scale  # noqa: E402

DEV = "cuda"
I0 = 1.0e4                       # photons per ray without an object
FILTERS = ("ramp", "hann", "cosine", "shepp-logan")


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # one slice looked at while the scan still runs: launches and latency count
        dict(name="fbp_preview", kind="fbp", slices=1, n=512, angles=360, operator="nearest", filter="hann",
             pad=2, offset=3.5),
        # a cropped detector: odd width, odd angle count, slices that fill no group of four or eight
        dict(name="fbp_odd", kind="fbp", slices=11, n=1001, angles=721, operator="nearest", filter="ramp",
             pad=1, offset=-2.25),
        # one pipeline chunk of the 2048^2 x 1800 volume this library is tuned on
        dict(name="fbp_volume", kind="fbp", slices=32, n=2048, angles=1800, operator="nearest", filter="hann",
             pad=2, offset=3.5),
        # the network's inputs: FBP with linear interpolation in FP32
        dict(name="fbp_linear", kind="fbp", slices=16, n=512, angles=720, operator="linear", filter="hann",
             pad=2, offset=0.0),
        # the same operator with the filtered rows stored as BF16
        dict(name="fbp_bf16", kind="fbp", slices=8, n=2048, angles=1800, operator="linear-bf16",
             filter="shepp-logan", pad=2, offset=3.5),
        # the drop-in call on a user's own numpy arrays, copies in and out inside
        dict(name="fbp_host", kind="fbp_host", slices=6, n=1024, angles=900, operator="nearest", filter="hamming",
             pad=2, offset=1.5),
        # simulated projections of a volume
        dict(name="radon", kind="radon", slices=24, n=1024, angles=900),
        # transmission EM on a block of a volume
        dict(name="tem", kind="tem", slices=16, n=1024, angles=900, iterations=3),
        # emission EM of a few small, odd-sized slices (fluorescence maps)
        dict(name="eem_small", kind="eem", slices=3, n=301, angles=257, iterations=10),
        # FBP by the slice theorem, the fast method for large volumes
        dict(name="bst", kind="bst", slices=8, n=2048, angles=1800, filter="ramp", pad=2),
        # transmission EM with the Fourier operators
        dict(name="temfq", kind="temfq", slices=6, n=1024, angles=900, pad=2, iterations=2),
        # one training step of the warm-start network
        dict(name="unet_train", kind="unet", slices=8, n=512),
    ]


def _updates(case):
    return case["slices"] * case["n"] ** 2 * case["angles"] * (1 + 2 * case.get("iterations", 0))


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fbp", "fbp", "fbp", "fbp_host", "radon", "tem", "eem", "bst", "temfq", "unet"])
    if kind == "unet":           # sides the network accepts: multiples of 8
        return dict(kind=kind, slices=rng.randint(1, 8), n=8 * _log_int(rng, 8, 64))
    n, angles, slices = _log_int(rng, 128, 2048), _log_int(rng, 90, 1800), _log_int(rng, 1, 32)
    c = dict(kind=kind, slices=slices, n=n, angles=angles)
    if kind in ("fbp", "fbp_host"):
        c.update(operator=rng.choice(["nearest", "nearest", "linear", "linear-bf16"]) if kind == "fbp" else "nearest",
                 pad=rng.choice([0, 1, 2, 2]), offset=round(rng.uniform(-4.0, 4.0), 2))
        c["filter"] = rng.choice(FILTERS[:3] if c["operator"] == "nearest" else FILTERS)
        if kind == "fbp_host":
            c.update(slices=min(slices, 8), n=min(n, 1400))
    elif kind in ("tem", "eem"):
        c.update(n=min(n, 1200), slices=min(slices, 16), iterations=rng.randint(2, 6))
    elif kind == "bst":          # even widths: the centre crop of the Fourier grid
        c.update(n=n - n % 2, slices=min(slices, 8), filter=rng.choice(FILTERS[:3]), pad=rng.choice([1, 2, 2]))
    elif kind == "temfq":
        c.update(n=min(n, 1024) - min(n, 1024) % 2, slices=min(slices, 6), pad=rng.choice([1, 2, 2]),
                 iterations=rng.randint(1, 3))
    # no larger than the listed cases: about a third of the largest one's updates
    c["slices"] = max(1, min(c["slices"], int(8e10 * c["slices"] / _updates(c))))
    return c


# ------------------------------------------------------------------ inputs --
def _ellipses(gen, slices, count):
    """[slices, count, 6] random ellipses inside the unit disc: x, y, half axes, angle, density."""
    u = torch.rand((slices, count, 6), generator=gen, device=DEV, dtype=torch.float64)
    a, b = 0.05 + 0.3 * u[..., 2], 0.05 + 0.3 * u[..., 3]
    r = torch.minimum(u[..., 0].sqrt(), (0.95 - torch.maximum(a, b)))
    phi = 2 * math.pi * u[..., 1]
    return torch.stack([r * phi.cos(), r * phi.sin(), a, b, math.pi * u[..., 4], u[..., 5]], -1)


def _projections(e, angles, t, sign):
    """Line integrals of the ellipses along x cos + sign y sin = t, [slices, angles, t], scaled to a maximum of 3."""
    th = torch.as_tensor(angles, dtype=torch.float32, device=DEV)[None, :, None]
    t = t[None, None, :].float()
    out = torch.zeros((e.shape[0], th.shape[1], t.shape[2]), device=DEV)
    for k in range(e.shape[1]):
        x, y, a, b, phi, rho = [v[:, None, None].float() for v in e[:, k].unbind(-1)]
        s2 = (a * torch.cos(th - sign * phi)) ** 2 + (b * torch.sin(th - sign * phi)) ** 2
        tau = t - (x * th.cos() + sign * y * th.sin())
        out += rho * 2 * a * b * (s2 - tau * tau).clamp(min=0).sqrt() / s2
    return out * (3.0 / out.amax((1, 2), keepdim=True))


def _counts(gen, p):
    return torch.poisson(I0 * torch.exp(-p), generator=gen).clamp(min=1.0)


def _images(gen, slices, n):
    e = _ellipses(gen, slices, 8)
    g = torch.linspace(-1, 1, n, device=DEV)
    img = torch.zeros((slices, n, n), device=DEV)
    for k in range(e.shape[1]):
        x, y, a, b, phi, rho = [v[:, None, None].float() for v in e[:, k].unbind(-1)]
        dx, dy = g[None, None, :] - x, g[None, :, None] - y
        u, v = dx * phi.cos() + dy * phi.sin(), dy * phi.cos() - dx * phi.sin()
        img += rho * ((u / a) ** 2 + (v / b) ** 2 <= 1)
    return img * (1 + 0.1 * torch.randn(img.shape, generator=gen, device=DEV))


def _angles(count):
    return (np.arange(count, dtype=np.float64) * (math.pi / count)).astype(np.float32)


def _ptr(a):
    return ctypes.c_void_p(a.data_ptr()) if torch.is_tensor(a) else a.ctypes.data_as(ctypes.c_void_p)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind, b, n = case["kind"], case["slices"], case["n"]
    s = dict(case=case)
    if kind == "unet":
        img = _images(gen, b, n)
        noise = torch.rand(img.shape, generator=gen, device=DEV)
        s.update(net=UNet.from_file(default_weights(), torch.device(DEV)), target=img, image=(img + 0.2 * noise).contiguous())
        s["scale"] = input_scale(s["image"])
        return s
    a = case["angles"]
    s["angles"] = _angles(a)
    if kind in ("fbp", "fbp_host", "bst"):
        t = (torch.arange(n, device=DEV, dtype=torch.float64) - n / 2) / (n / 2)
        sino = -torch.log(_counts(gen, _projections(_ellipses(gen, b, 12), s["angles"], t, -1)) / I0)
        s["ints"] = np.array([n, a, b, n, case["pad"], 0, 0, FilterNumber(case["filter"]), 0, 0], np.int32)
        s["floats"] = np.array([0, 0, 1, 0, 1, 1, case.get("offset", 0.0)], np.float32)
        if kind == "fbp_host":
            s["sino"] = sino.cpu().numpy()
            s["dic"] = {"gpu": [0], "angles[rad]": s["angles"], "filter": case["filter"], "padding": case["pad"],
                        "rotation axis offset": case["offset"]}
        else:
            s.update(sino=sino, image=torch.zeros((b, n, n), device=DEV))
    elif kind == "radon":
        s.update(image=_images(gen, b, n), sino=torch.zeros((b, a, n), device=DEV))
    else:
        t = torch.linspace(-1, 1, n, device=DEV, dtype=torch.float64)
        e = _ellipses(gen, b, 12)
        p = _projections(e, s["angles"], t, 1)
        s["image"] = torch.ones((b, n, n), device=DEV)
        if kind == "eem":
            s.update(data=_counts(gen, 3.0 - p) / I0 * 3.0, flat=None, start=1.0)
        elif kind == "tem":
            s.update(data=_counts(gen, p) / I0, flat=torch.ones((b, n), device=DEV), start=1.0)
        else:
            s.update(data=_counts(gen, p), flat=torch.full((b, n), I0, device=DEV))
            s["start"] = float(p.sum((1, 2)).mean()) * (2.0 / (n - 1)) / a / 4.0       # the mean density
            s["ints"] = np.array([n, a, b, n, case["pad"], 0, 0, b, case["iterations"], 1, 0], np.int32)
            s["floats"] = np.array([2.0 / (n - 1), 2.0 / (n - 1), 0], np.float32)
    return s


# --------------------------------------------------------------------- run --
def run(s):
    case = s["case"]
    kind, b, n = case["kind"], case["slices"], case["n"]
    if kind == "unet":
        # rate 0: the step runs whole and the state serves the next pass
        loss = s["net"].train_step(s["image"], s["target"], s["scale"], 0.0)
        return {"loss": loss, "weights": s["net"].gw, "biases": s["net"].gb}
    if kind == "fbp_host":
        return sscRaft.fbp(s["sino"], dic=dict(s["dic"]))
    a, ang = case["angles"], _ptr(s["angles"])
    if kind == "fbp":
        geometry, store = {"nearest": (0, 0), "linear": (1, 1), "linear-bf16": (1, 2)}[case["operator"]]
        rc = libraft.raft_fbp_device(0, _ptr(s["image"]), _ptr(s["sino"]), ang, _ptr(s["floats"]), _ptr(s["ints"]),
                                     geometry, store, _stream())
    elif kind == "bst":
        rc = libraft.raft_bst_device(0, _ptr(s["image"]), _ptr(s["sino"]), _ptr(s["floats"]), _ptr(s["ints"]),
                                     _stream())
    elif kind == "radon":
        rc = libraft.raft_radon_device(0, _ptr(s["sino"]), _ptr(s["image"]), ang, n, n, n, a, b, 1.0, 1.0, _stream())
    else:
        s["image"].fill_(s["start"])
        if kind == "temfq":
            rc = libraft.raft_temfq_device(0, _ptr(s["image"]), _ptr(s["data"]), _ptr(s["flat"]), ang,
                                           _ptr(s["floats"]), _ptr(s["ints"]), _stream())
        else:
            rc = libraft.raft_em_device(0 if kind == "tem" else 1, 0, _ptr(s["image"]), _ptr(s["data"]),
                                        _ptr(s["flat"]) if kind == "tem" else None, ang, n, a, b, case["iterations"],
                                        None, 1, _stream())
    if rc:
        check_error(kind)
    return s["sino"] if kind == "radon" else s["image"]


# -------------------------------------------------------------------- work --
def work(case):
    kind, b, n = case["kind"], case["slices"], case["n"]
    if kind == "unet":           # forward, data gradient (all but the first layer) and weight gradient
        side = {"0": n, "1": n // 2, "2": n // 4, "3": n // 8}
        conv = {l[0]: 2 * 9 * (1 if l[0] == "e0a" else l[1] + l[2]) * l[3] * side[l[0][1]] ** 2 for l in UNet.LAYERS}
        weights = sum(9 * (l[1] + l[2]) * l[3] for l in UNet.LAYERS)
        return {"bytes": 8 * b * n * n + 28 * weights, "flops": b * (3 * sum(conv.values()) - conv["e0a"])}
    a = case["angles"]
    grid, rows = b * n * n, b * a * n
    if kind in ("fbp", "fbp_host"):
        m = n * (1 + case["pad"])
        per = 1 if case["operator"] == "nearest" else 4      # an add; subtract, multiply-add and add
        return {"bytes": 4 * (grid + rows), "flops": b * a * 5 * m * math.log2(m) + per * grid * a}
    if kind == "bst":            # real transforms of the rows, half-rays, 2-D inverse transform
        m = n * (1 + case["pad"])
        return {"bytes": 4 * (grid + rows), "flops": b * math.log2(m) * (10 * a * m + 5 * m * m + 5 * m * n)}
    if kind == "radon":
        return {"bytes": 4 * (grid + rows), "flops": rows * n}
    it = case["iterations"]
    if kind in ("tem", "eem"):   # object and data, guess and result; the sensitivity image once
        return {"bytes": 4 * (2 * grid + rows), "flops": it * (rows * n + grid * a) + grid * a}
    m = n * (1 + case["pad"])
    project = b * math.log2(m) * (5 * m * n + 5 * m * m / 2 + 2.5 * m * a)
    back = b * (5 * a * m / 2 * math.log2(m) + 10 * n * n * math.log2(n))
    return {"bytes": 4 * (2 * grid + rows), "flops": it * (project + back) + back}


# --------------------------------------------------------------- tolerance --
def tolerance(case):
    """About four times the difference of two correct implementations (sums in
    another order, the other kernels of the library, or 64 bits)."""
    kind = case["kind"]
    if kind == "unet":           # BF16 activations through fourteen layers
        return {"rel": 1e-2}
    if case.get("operator") == "linear-bf16":
        return {"rel": 2e-3}
    return {"rel": 2e-5 if kind in ("tem", "eem") else 1e-5}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    kind = case["kind"]
    if kind != "unet" and _updates(case) > (7e10 if kind in ("bst", "temfq") else 1.5e11):
        return None
    s = prepare(case, seed)
    if kind == "unet":
        return _unet64(s)
    if kind in ("fbp", "fbp_host"):
        return _fbp64(s)
    if kind == "radon":
        return _project64(s["image"].double(), s["angles"], case["n"])
    if kind in ("tem", "eem"):
        return _em64(s)
    return _bst64(s) if kind == "bst" else _temfq64(s)


def _f32(x):
    """Rounds to single precision; the index rules are defined on single-precision positions."""
    return x.float().double()


def _steps(angles):
    d = np.diff(angles, append=angles[-1:])
    d[-1] = angles[-1] - angles[-2]
    return torch.as_tensor(d, device=DEV).double()


def _window(name, nu):
    """Apodisation of the ramp at nu = frequency / Nyquist."""
    return {"ramp": torch.ones_like(nu), "hann": 0.5 + 0.5 * torch.cos(math.pi * nu),
            "hamming": 0.54 + 0.46 * torch.cos(math.pi * nu), "cosine": torch.cos(0.5 * math.pi * nu),
            "shepp-logan": torch.sinc(0.5 * nu)}[name]


def _tent_window(name, w):
    """The nearest-sample operator's filters, on its weight w."""
    return {"ramp": torch.ones_like(w), "hann": 0.5 + 0.5 * torch.cos(2 * math.pi * w),
            "hamming": 0.54 + 0.46 * torch.cos(2 * math.pi * w), "cosine": torch.cos(0.5 * math.pi * w)}[name]


def _edge_pad(x, pad):
    n = x.shape[-1]
    i = (torch.arange(n * (1 + pad), device=DEV) - pad * n // 2).clamp(0, n - 1)
    return x[..., i]


def _fbp64(s):
    case = s["case"]
    n, pad, nearest = case["n"], case["pad"], case["operator"] == "nearest"
    m, off = n * (1 + pad), pad * n // 2
    k = torch.arange(m // 2 + 1, device=DEV).double()
    if nearest:
        h = m // 2 + 1
        w = 0.5 * torch.minimum(k, h - k) / h
        w, turn = w * _tent_window(case["filter"], w), case["offset"] * k / (2 * h - 2)
    else:
        w, turn = k / m * _window(case["filter"], 2 * k / m), case["offset"] * k / m
    spectrum = torch.polar(w / m, -2 * math.pi * turn)
    sino = torch.as_tensor(s["sino"], device=DEV)
    c32, s32 = np.cos(s["angles"]), np.sin(s["angles"])
    step = _steps(s["angles"])
    g = torch.arange(n, device=DEV).double() + off - m / 2
    out = torch.zeros((case["slices"], n * n), device=DEV, dtype=torch.float64)
    for a in range(case["angles"]):
        q = torch.fft.irfft(torch.fft.rfft(_edge_pad(sino[:, a].double(), pad)) * spectrum, n=m) * (m * step[a])
        if nearest:
            t = _f32(_f32(g[None, :] * float(c32[a]) - _f32(g * float(s32[a]))[:, None]) + m / 2).trunc().long()
            out += torch.where((t >= 0) & (t < m), q[:, t.clamp(0, m - 1)], 0.0).flatten(1)
        else:
            th = float(s["angles"][a])
            u = g[None, :] * math.cos(th) - g[:, None] * math.sin(th) + m / 2
            q, lo = tf.pad(q, (1, 1)), u.floor()
            i, f = lo.long().clamp(-1, m - 1) + 1, u - lo
            i, f = torch.where((lo < -1) | (lo >= m), torch.zeros_like(i), i), torch.where(lo < -1, 0.0, f)
            out += ((1 - f) * q[:, i] + f * q[:, (i + 1).clamp(max=m + 1)]).flatten(1)
    out = out.reshape(-1, n, n)
    return out.cpu().numpy() if case["kind"] == "fbp_host" else out


def _project64(img, angles, n):
    """Sum of the nearest pixels along each ray, rays and samples on [-1, 1]."""
    b = img.shape[0]
    d = float(np.float32(2.0 / (n - 1)))
    g = _f32(torch.arange(n, device=DEV).double() * d - 1)
    flat = tf.pad(img.reshape(b, -1), (0, 1))
    out = torch.zeros((b, len(angles), n), device=DEV, dtype=torch.float64)
    inv = float(np.float32(1.0) / np.float32(d))
    for a, th in enumerate(angles):
        c, si = float(np.cos(th)), float(np.sin(th))
        x = _f32(g[:, None] * c - _f32(g * si)[None, :])
        y = _f32(g[:, None] * si + _f32(g * c)[None, :])
        i, j = _f32(_f32(x + 1) * inv).trunc().long(), _f32(_f32(y + 1) * inv).trunc().long()
        inside = (i >= 0) & (i < n) & (j >= 0) & (j < n)
        out[:, a] = flat[:, torch.where(inside, j * n + i, n * n)].sum(-1) * d
    return out


def _back64(rows, angles, n):
    d = float(np.float32(2.0 / (n - 1)))
    g = _f32(torch.arange(n, device=DEV).double() * d - 1)
    inv = float(np.float32(1.0) / np.float32(d))
    step = _steps(angles)
    out = torch.zeros((rows.shape[0], n, n), device=DEV, dtype=torch.float64)
    for a, th in enumerate(angles):
        c, si = float(np.cos(th)), float(np.sin(th))
        t = _f32(_f32(_f32(g[None, :] * c + _f32(g * si)[:, None]) + 1) * inv).trunc().long()
        out += torch.where((t >= 0) & (t < n), rows[:, a][:, t.clamp(0, n - 1)], 0.0) * step[a]
    return out


def _em64(s):
    case, n = s["case"], s["case"]["n"]
    data = s["data"].double()
    tem = case["kind"] == "tem"
    norm = _back64(data if tem else torch.ones_like(data), s["angles"], n)
    x = torch.full_like(norm, s["start"])
    for _ in range(case["iterations"]):
        p = _project64(x, s["angles"], n)
        if tem:
            q = s["flat"].double()[:, None, :] * torch.exp(-p)
        else:
            q = (data * torch.sign(p) / torch.sqrt(1e-8 + p * p)).clamp(min=0)
        x = x * _back64(q, s["angles"], n) / norm
    return x


def _polar_to_image64(rows, length, grid, off, n, weight, scale):
    """Inverse of the slice theorem: half-rays [angles, samples] of one slice to an n x n image."""
    a, width = rows.shape
    half = width // 2
    w = torch.full((half,), weight, device=DEV, dtype=torch.float64)
    w[0] *= 0.5
    rays = torch.cat([rows[:, :half].flip(-1), rows[:, half:2 * half]]) * w
    k = torch.arange(length, device=DEV).double()
    m = torch.minimum(k, length - k).clamp(min=0.5)
    polar = torch.fft.fft(tf.pad(rays, (0, length - half))) * (2 / (length * m))
    i = torch.arange(grid, device=DEV)
    px, py = (i - grid // 2).float()[None, :], (i - grid // 2).float()[:, None]
    rho = length * torch.hypot(px, py) / grid
    arc = 2 * a * (0.5 * torch.atan2(py, px) / np.float32(math.pi) + 0.5)
    ir, ia = rho.long(), arc.long()
    f, t = (rho - ir).double(), (ia - arc).double()
    inside = ir < length // 2 - 1
    ir = torch.where(inside, ir, 0)
    lo, hi = (ia % (2 * a)) * length, ((ia + 1) % (2 * a)) * length
    polar = polar.flatten()
    v = t * ((1 - f) * polar[lo + ir] + f * polar[lo + ir + 1])
    v += (1 - t) * ((1 - f) * polar[hi + ir] + f * polar[hi + ir + 1])
    sign = 1.0 - 2.0 * ((i % 2)[None, :] != (i % 2)[:, None])
    v = torch.where(inside, v, 0.0) * sign
    v = torch.roll(v, (grid // 2, grid // 2), (0, 1))
    return torch.fft.ifft2(v, norm="forward").real[off:off + n, off:off + n] / scale


def _bst64(s):
    case = s["case"]
    n, pad = case["n"], case["pad"]
    m, off = n * (1 + pad), pad * n // 2
    k = torch.arange(m, device=DEV).double()
    w = torch.minimum(k, m - k) / m
    w = w * _tent_window(case["filter"], w)
    out = torch.empty((case["slices"], n, n), device=DEV, dtype=torch.float64)
    for z in range(case["slices"]):
        rows = torch.fft.ifft(torch.fft.fft(_edge_pad(s["sino"][z].double(), pad)) * w, norm="forward").real
        out[z] = _polar_to_image64(rows, m, m, off, n, 4.0, 4.0 * m)
    return out


def _temfq64(s):
    case = s["case"]
    n, a, pad = case["n"], case["angles"], case["pad"]
    m, lb = n * (1 + pad), n * (1 + pad) // 2
    scale = float(np.float32(s["floats"][0]) / np.float32(m))
    c32 = torch.as_tensor(np.cos(s["angles"]), device=DEV)[:, None]
    s32 = torch.as_tensor(np.sin(s["angles"]), device=DEV)[:, None]
    rho = (torch.arange(m, device=DEV) - m // 2).float()[None, :]
    x, y = c32 * rho, s32 * rho
    x0, y0 = x.floor(), y.floor()
    fx, fy = (x - x0).double(), (y - y0).double()

    def back(rows):
        return _polar_to_image64(rows, lb, n, 0, n, float((1 + pad) ** 2), 1.0)

    def at(spec, i, j):
        return spec[(j.long() + m // 2) % m, (i.long() + m // 2) % m]

    def forward(img, flat):
        lead = (m - n) // 2
        big = tf.pad(img, (lead, m - n - lead, lead, m - n - lead))
        spec = torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(big)))
        v = (1 - fy) * ((1 - fx) * at(spec, x0, y0) + fx * at(spec, x0 + 1, y0))
        v += fy * ((1 - fx) * at(spec, x0, y0 + 1) + fx * at(spec, x0 + 1, y0 + 1))
        p = torch.fft.fftshift(torch.fft.ifft(torch.fft.ifftshift(v, dim=-1), norm="forward"), dim=-1)
        p = p.real[:, lead:lead + n] * scale
        return flat * torch.exp(-p.clamp(min=0))

    out = torch.empty((case["slices"], n, n), device=DEV, dtype=torch.float64)
    for z in range(case["slices"]):
        norm = back(s["data"][z].double())
        img = torch.full_like(norm, float(np.float32(s["start"])))
        for _ in range(case["iterations"]):
            img = img * back(forward(img, s["flat"][z].double())) / norm
        out[z] = img
    return out


def _unet64(s):
    net = s["net"]
    w = {k: net.wb[k].double().permute(0, 3, 1, 2).requires_grad_() if k in net.wb
         else net.w[k].double().requires_grad_() for k in net.w}
    bias = {k: v.double().requires_grad_() for k, v in net.b.items()}

    def conv(k, x):
        # shifted products: a 64-bit convolution of a library may be slow
        n, c, h, wd = x.shape
        x, out = tf.pad(x, (1, 1, 1, 1)), bias[k][None, :, None, None]
        for dy in range(3):
            for dx in range(3):
                tap = x[:, :, dy:dy + h, dx:dx + wd]
                out = out + torch.einsum("nchw,oc->nohw", tap, w[k][:, :c, dy, dx])
        return torch.relu(out)

    def up(x):
        return tf.interpolate(x, scale_factor=2, mode="nearest")

    names = list(w)
    loss = torch.zeros((), device=DEV, dtype=torch.float64)
    grads = {k: 0.0 for k in names}, {k: 0.0 for k in names}
    total = s["image"].numel()
    for z in range(s["image"].shape[0]):
        x = (s["image"][z] * s["scale"][z]).double()[None, None]
        e0 = conv("e0b", conv("e0a", x.bfloat16().double()))
        e1 = conv("e1b", conv("e1a", tf.avg_pool2d(e0, 2)))
        e2 = conv("e2b", conv("e2a", tf.avg_pool2d(e1, 2)))
        e3 = conv("e3b", conv("e3a", tf.avg_pool2d(e2, 2)))
        d2 = conv("d2b", conv("d2a", torch.cat([up(e3), e2], 1)))
        d1 = conv("d1b", conv("d1a", torch.cat([up(d2), e1], 1)))
        d0 = conv("d0b", conv("d0a", torch.cat([up(d1), e0], 1)))
        out = torch.einsum("nchw,c->nhw", d0, w["head"]) + bias["head"] + x[:, 0]
        one = ((out - (s["target"][z] * s["scale"][z]).double()) ** 2).sum() / total
        got = torch.autograd.grad(one, [w[k] for k in names] + [bias[k] for k in names])
        loss += one.detach()
        for i, k in enumerate(names):
            grads[0][k] = grads[0][k] + got[i]
            grads[1][k] = grads[1][k] + got[len(names) + i]
    weights = {k: (g.permute(0, 2, 3, 1) if g.dim() == 4 else g) for k, g in grads[0].items()}
    return {"loss": loss[None], "weights": weights, "biases": grads[1]}
