"""Performance cases of the scattering engine: whole requests through the public
entry points, over the sizes, data types and options users run.

Sizes and physics are those of the repository's workloads
(cyrsoxs_gb300/workloads.py: the first configuration, the batched set, the
serving stream, the 256 x 512 x 512 request) and of its parity tests (frames,
interpolation, windows, tilted k, 2D, FP64).  A case is a dict:

  kind        device   simulate_device: morphology and patterns on the GPU
              host     cuda_main: numpy arrays in and out, as the drop-in is called
              fp64     simulate_device_fp64 on float4 voxels
              served   the serving engine over a set of uneven requests
  nx, ny, nz  voxels; materials, energies (count), angles (count, `step` degrees)
  phys        voxel size in nm; morphology euler | vector; interp linear | nearest
  window, mask, frame (lab | material), tilted (two tilted k vectors instead of z)

Inputs are seeded: smooth random phases and director fields, uniform order
parameter, Lorentzian optical constants.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cyrsoxs_gb300 import _native, serving

_BASE = dict(kind="device", materials=2, energies=10, angles=12, step=15.0, phys=5.0, morphology="euler",
             interp="linear", window=False, mask=False, frame="lab", tilted=False, requests=1)


def _case(nx, ny, nz, **over):
    return dict(_BASE, nx=nx, ny=ny, nz=nz, **over)


def listed():
    return [
        # the smallest request a user sends (a test-sized volume, two energies): latency and launches
        dict(_case(64, 64, 16, energies=2, angles=6, step=30.0), name="small_request"),
        # the first configuration: 32 x 256 x 256, 3 energies x 12 angles
        dict(_case(256, 256, 32, energies=3), name="first_config"),
        # the batched set: uneven small morphologies queued together on the serving engine
        dict(_case(256, 256, 64, kind="served", energies=20, requests=12), name="served_set"),
        # a serving-stream request with FFT-friendly lengths that are not powers of two
        dict(_case(240, 240, 90, materials=3, energies=24, angles=18, step=10.0, phys=2.0), name="ragged_smooth"),
        # the share of the serving stream whose lengths are arbitrary (prime factors above 7 on every axis)
        dict(_case(211, 211, 61, energies=16, angles=10, phys=2.0), name="ragged_prime"),
        # one energy, windowed: an alignment run before a full energy scan (the spectra are formed per energy)
        dict(_case(256, 256, 128, materials=4, energies=1, angles=36, step=5.0, phys=2.0, window=True),
             name="single_energy"),
        # vector morphology in the material frame with nearest-neighbour sampling and the rotation mask
        dict(_case(128, 128, 64, materials=3, energies=10, morphology="vector", interp="nearest", mask=True,
                   frame="material"), name="material_frame"),
        # beam divergence: two tilted k vectors, all six tensor entries
        dict(_case(256, 256, 64, energies=8, phys=2.0, tilted=True, mask=True), name="beam_divergence"),
        # a thin film as one plane, 1024 x 1024 detector
        dict(_case(1024, 1024, 1, materials=3, energies=20, angles=36, step=5.0, phys=2.0), name="film_2d"),
        # the drop-in call of a Python user: numpy arrays through cuda_main, copies included
        dict(_case(256, 256, 64, kind="host", energies=10), name="host_call"),
        # the double-precision build's workload, on the first configuration
        dict(_case(256, 256, 32, kind="fp64", energies=3), name="fp64_request"),
        # the benchmark request: 256 x 512 x 512, 4 materials, 50 energies x 36 angles
        dict(_case(512, 512, 256, materials=4, energies=50, angles=36, step=5.0, phys=2.0), name="full_scan"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """An axis length in [lo, hi]: a power of two, a 7-smooth length, or any length."""
    how = rng.random()
    n = _log_int(rng, lo, hi)
    if how < 0.4:
        return max(lo, min(hi, 2 ** round(math.log2(n))))
    if how < 0.8:
        def smooth(v):
            for p in (2, 3, 5, 7):
                while v % p == 0:
                    v //= p
            return v == 1
        while not smooth(n) and n > lo:
            n -= 1
    return n


def draw(rng):
    kind = rng.choice(["device"] * 7 + ["fp64", "host", "served"])
    step = rng.choice([5.0, 7.5, 10.0, 15.0, 30.0])
    common = dict(kind=kind, angles=rng.randint(max(1, int(60 / step)), int(180 / step)), step=step,
                  phys=rng.choice([2.0, 2.0, 5.0]), morphology=rng.choice(["euler", "euler", "vector"]))
    if kind == "served":
        xy = rng.choice([64, 96, 128, 256])
        return _case(xy, xy, rng.choice([16, 32, 64]), **dict(common, energies=rng.randint(4, 20),
                                                              requests=rng.randint(4, 12)))
    if kind == "fp64":
        nx = _length(rng, 40, 256)
        ny, nz, m, ne = (nx if rng.random() < 0.7 else _length(rng, 40, 256)), _length(rng, 8, 32), rng.randint(1, 3), rng.randint(1, 4)
    else:
        nx = _length(rng, 48, 512)
        ny = nx if rng.random() < 0.8 else _length(rng, 48, 512)
        nz = 1 if rng.random() < 0.1 else _length(rng, 8, 128)
        m, ne = rng.randint(1, 4), _log_int(rng, 1, 50)
    more = dict(interp=rng.choice(["linear", "linear", "nearest"]), window=rng.random() < 0.2, mask=rng.random() < 0.4,
                frame="material" if rng.random() < 0.15 else "lab", tilted=rng.random() < 0.15)
    if more["frame"] == "material" or more["tilted"]:
        ne = min(ne, 10)
    return _case(nx, ny, nz, **dict(common, **more, materials=m, energies=ne))


# --------------------------------------------------------------------------- inputs


def _requests(case):
    """The single requests of a case: itself, or the uneven sizes of a served set (X = Y halved and Z varied)."""
    if case["kind"] != "served":
        return [case]
    out = []
    for i in range(case["requests"]):
        xy = max(32, case["nx"] >> (i % 3))
        out.append(dict(case, kind="device", nx=xy, ny=xy, nz=max(16, case["nz"] >> ((i // 3) % 3))))
    return out


def _energies(case):
    n = case["energies"]
    return np.linspace(270.0, 300.0, n).astype(np.float32) if n > 1 else np.array([285.0], np.float32)


def _k_vectors(case):
    ks = [[0.05, 0.02, 1.0], [-0.04, 0.03, 1.0]] if case["tilted"] else [[0.0, 0.0, 1.0]]
    return np.stack([(np.array(k) / np.linalg.norm(k)).astype(np.float32) for k in ks])


def _optical(case, seed):
    """[E][M][4] (delta_par, beta_par, delta_perp, beta_perp): two Lorentzian resonances per material."""
    rng = np.random.default_rng(seed + 17)
    e = _energies(case).astype(np.float64)
    out = np.zeros((len(e), case["materials"], 4))
    for m in range(case["materials"]):
        e0, amp, wid = rng.uniform(278, 292, 2), rng.uniform(2e-3, 8e-3, 2), rng.uniform(0.5, 2.0, 2)
        lor = sum(a / (1 + ((e - c) / (0.5 * w)) ** 2) for a, c, w in zip(amp, e0, wid))
        base, aniso = 1e-3 * (1 + 0.2 * m), rng.uniform(0.3, 0.9)
        out[:, m] = np.stack([base + lor, 0.4 * base + 0.5 * lor, base + aniso * lor,
                              0.4 * base + 0.5 * aniso * lor], -1)
    return out.astype(np.float32)


def _smooth(g, shape, width):
    f = torch.randn(shape, generator=g, device="cuda")[None, None]
    for axis in range(3):
        if shape[axis] < width:
            continue
        k = [1, 1, 1]
        k[axis] = width
        pad = [v // 2 for v in k]
        f = torch.nn.functional.avg_pool3d(f, k, stride=1, padding=pad, count_include_pad=False)
    return f[0, 0]


def _voxels(case, seed):
    """[M][Z][Y][X][4] float32 on the GPU: Euler (S, theta, psi, Vfrac) or vector (sx, sy, sz, phi_unaligned)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    out = torch.empty((case["materials"], *shape, 4), device="cuda")
    total = torch.zeros(shape, device="cuda")
    for m in range(case["materials"]):
        f = _smooth(g, shape, 7)
        f = torch.exp(f.mul_(4.0 / (float(f.std()) + 1e-12)))
        out[m, ..., 3] = f
        total += f
    out[..., 3] /= total
    for m in range(case["materials"]):
        order = torch.rand(shape, generator=g, device="cuda")
        n = torch.stack([_smooth(g, shape, 5) for _ in range(3)], -1)
        n /= n.norm(dim=-1, keepdim=True).clamp_min(1e-12)
        if case["morphology"] == "euler":
            out[m, ..., 0] = order
            out[m, ..., 1] = torch.acos(n[..., 2].clamp(-1, 1))
            out[m, ..., 2] = torch.atan2(n[..., 1], n[..., 0]) % (2 * math.pi)
        else:
            aligned = out[m, ..., 3] * order
            out[m, ..., :3] = aligned.sqrt()[..., None] * n
            out[m, ..., 3] -= aligned
    return out


def _options(case):
    return _native.Options(nx=case["nx"], ny=case["ny"], nz=case["nz"], num_material=case["materials"],
                           energies=_energies(case), start_angle=0.0,
                           end_angle=case["step"] * (case["angles"] - 1), increment_angle=case["step"],
                           phys_size=case["phys"], case_type=1 if case["tilted"] else 0, k_vectors=_k_vectors(case),
                           morphology_type=0 if case["morphology"] == "euler" else 1,
                           ewald_interpolation=1 if case["interp"] == "linear" else 0,
                           windowing=int(case["window"]), rot_mask=int(case["mask"]),
                           reference_frame=1 if case["frame"] == "lab" else 0)


def _one(case, seed):
    opts, optical, vox = _options(case), _optical(case, seed), _voxels(case, seed)
    shape = (case["energies"], opts.num_k, case["ny"], case["nx"])
    if case["kind"] == "host":
        return dict(opts=opts, optical=optical, vox=vox.cpu().numpy(), out=np.zeros(shape, np.float32))
    dtype = torch.float64 if case["kind"] == "fp64" else torch.float32
    if case["kind"] == "fp64":
        optical = optical.astype(np.float64)
    return dict(opts=opts, optical=optical, vox=vox, out=torch.zeros(shape, dtype=dtype, device="cuda"))


def prepare(case, seed):
    state = dict(kind=case["kind"], requests=[_one(c, seed + 1000 * i) for i, c in enumerate(_requests(case))])
    if case["kind"] == "served":
        state["server"] = serving.Server(slots=8, graphs=True, groups=True)
    return state


def run(state):
    reqs = state["requests"]
    if state["kind"] == "served":
        ids = [state["server"].submit(r["opts"], r["optical"], r["vox"].data_ptr(), r["out"].data_ptr(), device=True)
               for r in reqs]
        for i in ids:
            state["server"].wait(i)
        return [r["out"] for r in reqs]
    r = reqs[0]
    if state["kind"] == "host":
        return _native.cuda_main(r["opts"], r["optical"], r["vox"], out=r["out"])
    stream = torch.cuda.current_stream().cuda_stream
    if state["kind"] == "fp64":
        _native.simulate_device_fp64(r["opts"], r["optical"], r["vox"].data_ptr(), False, r["out"].data_ptr(), stream)
    else:
        _native.simulate_device(r["opts"], r["optical"], r["vox"].data_ptr(), r["out"].data_ptr(), stream)
    return r["out"]


def work(case):
    """Voxels and constants read once, patterns written once; the transforms of the 7 M + 1 real fields of
    the morphology, their combination at two Ewald planes per pixel, energy and k, and one bilinear sample
    per pixel, energy, k and angle."""
    nbytes, flops = 0, 0
    for c in _requests(case):
        vox, pix = c["nx"] * c["ny"] * c["nz"], c["nx"] * c["ny"] * c["energies"] * (2 if c["tilted"] else 1)
        fields = 7 * c["materials"] + 1
        item = 8 if c["kind"] == "fp64" else 4
        nbytes += 16 * vox * c["materials"] + item * pix + 16 * c["energies"] * c["materials"]
        flops += vox * (2.5 * fields * math.log2(vox) + 40 * c["materials"])
        flops += pix * (2 * (8 * fields + 60) + 20 * c["angles"])
    return {"bytes": float(nbytes), "flops": float(flops)}


# --------------------------------------------------------------------------- the same patterns in 64 bits
#
# The amplitudes are doubles.  Which pixel is a number, which Ewald planes it takes and where a rotated
# pixel samples its source are decided in float32, as the entry points define them.

_F = np.float32


def _cross(a, b):
    return np.array([a[1] * b[2] - a[2] * b[1], -(a[0] * b[2] - a[2] * b[0]), a[0] * b[1] - a[1] * b[0]], _F)


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _matmul(a, b):
    r = np.zeros((3, 3), _F)
    for i in range(3):
        for j in range(3):
            for k in range(3):
                r[i, j] = r[i, j] + a[i, k] * b[k, j]
    return r


def _inverse(a):
    det = float(a[0, 0] * (a[1, 1] * a[2, 2] - a[2, 1] * a[1, 2]) - a[0, 1] * (a[1, 0] * a[2, 2] - a[1, 2] * a[2, 0])
                + a[0, 2] * (a[1, 0] * a[2, 1] - a[1, 1] * a[2, 0]))
    adj = [[a[1, 1] * a[2, 2] - a[2, 1] * a[1, 2], a[0, 2] * a[2, 1] - a[0, 1] * a[2, 2], a[0, 1] * a[1, 2] - a[0, 2] * a[1, 1]],
           [a[1, 2] * a[2, 0] - a[1, 0] * a[2, 2], a[0, 0] * a[2, 2] - a[0, 2] * a[2, 0], a[1, 0] * a[0, 2] - a[0, 0] * a[1, 2]],
           [a[1, 0] * a[2, 1] - a[2, 0] * a[1, 1], a[2, 0] * a[0, 1] - a[0, 0] * a[2, 1], a[0, 0] * a[1, 1] - a[1, 0] * a[0, 1]]]
    return np.array(adj, _F) * _F(1.0 / det)


def _between(a, b):
    """Rotation taking unit vector a onto b."""
    if np.all(np.abs(a - b) < 1e-6):
        return np.eye(3, dtype=_F)
    c, ax = _dot(a, b), _cross(a, b)
    s = np.sqrt(_dot(ax, ax))
    rej = b - c * a
    rot = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]], _F)
    frame = np.stack([a, rej / np.sqrt(_dot(rej, rej)), -ax], 1)
    return _matmul(frame, _matmul(rot, _inverse(frame)))


def _about(v, axis, angle):
    """v turned about axis by each of the angles: [3, n] float32."""
    angle = np.atleast_1d(np.asarray(angle, _F)).astype(np.float64)
    c, s = np.cos(angle).astype(_F), np.sin(angle).astype(_F)
    cr, k = _cross(axis, v), (_F(1) - c) * _dot(axis, v)
    return np.stack([c * v[i] + s * cr[i] + k * axis[i] for i in range(3)])


def _warp(c):
    """Sample coefficients (float32) of the affine map c (source to destination, double)."""
    det = c[0][0] * c[1][1] - c[0][1] * c[1][0]
    a = [_F(c[1][1] / det), _F(-c[0][1] / det), _F(-c[1][0] / det), _F(c[0][0] / det)]
    offs = [_F(-(float(a[2 * i]) * c[0][2] + float(a[2 * i + 1]) * c[1][2])) for i in range(2)]
    return a[0], a[1], offs[0], a[2], a[3], offs[1]


def _sample(img, w, h, coef, fill):
    """Bilinear samples of img [h, w] at every destination pixel; `fill` where the source lies outside."""
    x = torch.arange(w, device=img.device, dtype=torch.float64)[None, :]
    y = torch.arange(h, device=img.device, dtype=torch.float32)[:, None]

    def position(a, b, off):
        by = y * torch.tensor(float(b), dtype=torch.float32, device=img.device)
        return (float(a) * x + by.double()).float() + torch.tensor(float(off), dtype=torch.float32, device=img.device)

    xs, ys = position(*coef[:3]), position(*coef[3:])
    inside = (xs >= 0) & (xs <= w - 1) & (ys >= 0) & (ys <= h - 1)
    xs, ys = torch.where(inside, xs, 0), torch.where(inside, ys, 0)
    x0, y0 = xs.floor().long().clamp_max(w - 1), ys.floor().long().clamp_max(h - 1)
    x1, y1 = (x0 + 1).clamp_max(w - 1), (y0 + 1).clamp_max(h - 1)
    fx, fy = (xs - x0.float()).double(), (ys - y0.float()).double()
    flat = img.reshape(-1)
    top = (1 - fx) * flat[y0 * w + x0] + fx * flat[y0 * w + x1]
    low = (1 - fx) * flat[y1 * w + x0] + fx * flat[y1 * w + x1]
    return torch.where(inside, (1 - fy) * top + fy * low, fill)


def _spectra(case, vox):
    """[M][7] transforms (complex128, flat) of u_x^2 u_y^2 u_z^2 u_x u_y u_x u_z u_y u_z phi_ui, windowed,
    bin 0 replaced by the mean of its neighbours."""
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    win = 1.0
    if case["window"]:
        for axis, n in enumerate((nz, ny, nx)):
            h = 0.5 * (1 - torch.cos(2 * math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n))
            if n > 1:
                win = win * h.view([n if a == axis else 1 for a in range(3)])
    out = []
    for m in range(case["materials"]):
        s = [vox[m, ..., i].double() for i in range(4)]
        if case["morphology"] == "euler":
            aligned = s[0] * s[3]
            n = (s[2].cos() * s[1].sin(), s[2].sin() * s[1].sin(), s[1].cos())
            free = s[3] - aligned
        else:
            aligned, n, free = 1.0, s[:3], s[3]
        row = []
        for f in (n[0] * n[0], n[1] * n[1], n[2] * n[2], n[0] * n[1], n[0] * n[2], n[1] * n[2], None):
            f = torch.fft.fftn((free if f is None else aligned * f) * win)
            near = [f[0, 0, 1], f[0, 1 % ny, 0], f[0, 0, nx - 1], f[0, ny - 1, 0]]
            if nz > 1:
                near += [f[1, 0, 0], f[nz - 1, 0, 0]]
            f[0, 0, 0] = sum(near) / len(near)
            row.append(f.reshape(-1))
        out.append(row)
    return out


def _planes(case, kmag, k):
    """Per pixel [ny, nx]: whether it is a number, its Ewald planes and the second one's weight (float32 rules)."""
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    q = 2.0 * math.pi / case["phys"]
    start = _F(-_F(math.pi / case["phys"]))
    d = [_F(q / (n - 1)) if n > 1 else _F(0) for n in (nx, ny, nz)]
    kv = [_F(kmag * c) for c in k]
    ax = kv[0] + (start + np.arange(nx, dtype=_F) * d[0])
    ay = kv[1] + (start + np.arange(ny, dtype=_F) * d[1])
    val = (kmag * kmag - (ax * ax)[None, :]) - (ay * ay)[:, None]
    ok = val >= 0
    ok[:, nx - 1] = False
    ok[ny - 1, :] = False
    z0 = np.zeros((ny, nx), np.int64)
    w1 = np.zeros((ny, nx))
    two = nz > 1 and case["interp"] == "linear"
    if nz > 1:
        pos = -kv[2] + np.sqrt(np.where(ok, val, 0).astype(_F))
        t = (pos - start) / d[2]
        if two:
            z0 = np.where(t <= 0, 0, t).astype(np.int64)
            ok &= z0 < nz - 1
            w1 = (pos.astype(np.float64) - (float(start) + (z0.astype(_F) * d[2]).astype(np.float64))) / float(d[2])
        else:
            z0 = np.where(t <= 0, 0, np.floor(np.abs(t.astype(np.float64)) + 0.5)).astype(np.int64)
            ok &= z0 <= nz - 1
    z0 = np.where(ok, z0, 0)
    qs = [((-math.pi / case["phys"]) + (np.arange(n, dtype=_F) * dd).astype(np.float64)).astype(_F)
          for n, dd in zip((nx, ny, nz), d)]
    if nz == 1:
        qs[2] = np.zeros(1, _F)
    return ok, z0, w1, two, kv, qs


def _shift(j, n):
    return (n // 2 - j) % n


def _patterns(case, seed):
    vox = _voxels(case, seed)
    spec = _spectra(case, vox)
    del vox
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    optical = _optical(case, seed).astype(np.float64)
    dev, nan = "cuda", float("nan")
    on = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
    out = torch.empty((case["energies"], len(_k_vectors(case)), ny, nx), dtype=torch.float64, device=dev)
    eye = np.array([0, 0, 1], _F)
    frames = []
    for k in _k_vectors(case):
        rk = _between(eye, k)
        sx = rk[:, 0].copy()
        steps = np.arange(100000, dtype=_F) * _F(math.pi / 100000)
        at = steps[np.argmin(np.abs(_about(sx, k, steps)[1]))]
        base = at if _about(sx, k, at)[0, 0] > 0 else _F(float(at) + math.pi)
        turns = []
        for i in range(case["angles"]):
            ang = _F(float(base + _F(0) + _F(i) * _F(case["step"])) * math.pi / 180.0)
            r = _matmul(_between(sx, _about(sx, k, ang)[:, 0]), rk)
            a, b = float(_F(math.cos(ang))), float(_F(math.sin(ang)))
            c = [[a, b, float(_F((1 - a) * nx / 2 - b * ny / 2.0))], [-b, a, float(_F(b * nx / 2.0 + (1 - a) * ny / 2.0))]]
            turns.append((r.astype(np.float64), _warp(c)))
        # the detector's image of the three reference points under R_k
        sp = [(nx / 2.0, ny / 2.0), (nx * 0.5, ny * 1.0), (nx * 1.0, ny * 0.5)]
        dp = []
        for px, py in sp:
            s = np.array([px - nx / 2.0, py - ny / 2.0, 0.0], _F)
            dp.append([float(_F(float(rk[i, 0] * s[0] + rk[i, 1] * s[1] + rk[i, 2] * s[2]) + (nx, ny)[i] / 2.0)) for i in range(2)])
        (x0, y0), (x1, y1), (x2, y2) = sp
        den = x0 * y1 - x1 * y0 - x0 * y2 + x2 * y0 + x1 * y2 - x2 * y1
        det = []
        for i in range(2):
            u0, u1, u2 = (p[i] for p in dp)
            det.append([(u0 * y1 - u1 * y0 - u0 * y2 + u2 * y0 + u1 * y2 - u2 * y1) / den,
                        -(u0 * x1 - u1 * x0 - u0 * x2 + u2 * x0 + u1 * x2 - u2 * x1) / den,
                        (u0 * x1 * y2 - u0 * x2 * y1 - u1 * x0 * y2 + u1 * x2 * y0 + u2 * x0 * y1 - u2 * x1 * y0) / den])
        frames.append((k, turns, _warp(det)))
    ux, uy = on(_shift(np.arange(nx), nx))[None, :], on(_shift(np.arange(ny), ny))[:, None]
    sym = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
    for e, energy in enumerate(_energies(case)):
        kmag = _F(2 * math.pi / float(_F(1239.84197 / float(energy))))
        par, per = 1.0 - optical[e, :, 0] + 1j * optical[e, :, 1], 1.0 - optical[e, :, 2] + 1j * optical[e, :, 3]
        s = 0.25 / math.pi
        # contrasts n^2 - 1 of the aligned fraction along and across the director, and of the unaligned one
        A, B = s * (par * par - 1), s * (per * per - 1)
        C = s * (((par + 2 * per) / 3) ** 2 - 1)
        for ki, (k, turns, det) in enumerate(frames):
            ok, z0, w1, two, kv, qs = _planes(case, kmag, k)
            ok, z0, w1 = on(ok), on(z0), on(w1)
            fields = []
            for p in range(2 if two else 1):
                z = (nz // 2 - (z0 + p)) % nz
                idx = (z * ny + uy) * nx + ux
                nt = [0.0] * 6
                for m in range(case["materials"]):
                    g = [f[idx] for f in spec[m]]
                    tr = g[0] + g[1] + g[2]
                    for v, f in ((0, 0), (3, 1), (5, 2)):
                        nt[v] = nt[v] + complex(A[m] - B[m]) * g[f] + complex(B[m]) * tr + complex(C[m]) * g[6]
                    for v, f in ((1, 3), (2, 4), (4, 5)):
                        nt[v] = nt[v] + complex(A[m] - B[m]) * g[f]
                Q = [float(kv[0]) + on(qs[0]).double()[None, :], float(kv[1]) + on(qs[1]).double()[:, None],
                     float(kv[2]) + on(qs[2]).double()[(z0 + p).clamp_max(nz - 1)]]
                fields.append((nt, Q))
            total = torch.zeros((nx, ny), dtype=torch.float64, device=dev)
            count = torch.zeros((nx, ny), dtype=torch.float64, device=dev)
            for r, coef in turns:
                inten = []
                for nt, Q in fields:
                    pol = [sum(float(r[b, 0]) * nt[sym[c][b]] for b in range(3)) for c in range(3)]
                    if case["frame"] == "material":
                        pol = [sum(float(r[c, a]) * pol[c] for c in range(3)) for a in range(3)]
                    qp = sum(Q[c] * pol[c] for c in range(3))
                    amp = [float(kmag) ** 2 * pol[c] - Q[c] * qp for c in range(3)]
                    inten.append(sum(t.real * t.real + t.imag * t.imag for t in amp))
                img = (1 - w1) * inten[0] + w1 * inten[1] if two else inten[0]
                img = torch.where(ok, img, nan)
                # the rotation sees the same buffer as an image of width ny and height nx
                v = _sample(img.reshape(nx, ny), ny, nx, coef, nan)
                if case["mask"]:
                    seen = ~torch.isnan(v)
                    total += torch.where(seen, v, 0.0)
                    count += seen
                else:
                    total += v
            mean = torch.where(count > 0, total / count.clamp_min(1), 0.0) if case["mask"] else total / len(turns)
            out[e, ki] = _sample(mean, ny, nx, det, 0.0 if case["mask"] else nan).reshape(ny, nx)
    return out


def exact(case, seed):
    got = [_patterns(c, seed + 1000 * i) for i, c in enumerate(_requests(case))]
    if case["kind"] == "served":
        return got
    return got[0].cpu().numpy() if case["kind"] == "host" else got[0]
