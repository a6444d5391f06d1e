"""Measured cases: what users of the library have it do, through its public
entry points, from single small calls to full-size reconstructions.

A case is a dict of plain values:

  op       project | backproject | pair | two | host | grad | attgrad | osem | batch
  nx ny nz grid (arrays are (nz, ny, nx), x fastest)
  ncam     cameras, equispaced over `arc` degrees about the gantry axis
  arc      360 (opposite cameras present) or 180 (a cardiac half-turn)
  tilt     degrees about the other two axes; 0 keeps the cameras on the gantry
  psf      width of the depth-dependent PSF (0: none)
  att      attenuation map present
  dtype    storage of activity and mu: f32 | bf16 | f64
  subsets  OSEM subsets (osem)
  volumes, first, trim   mix of the batched reconstruction (batch)

Volumes are seeded ellipsoid phantoms, sinograms Poisson counts of a plain
projection of the phantom.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from niftyrec_gb300 import _lib, array_api, autograd, precision
from niftyrec_gb300.batch import Batch
from niftyrec_gb300.plan import Plan

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f64": torch.float64}
EPSILON = 1e-6


def _case(op, nx, ny, nz, ncam, psf=0, att=True, dtype="f32", arc=360, tilt=0.0, **more):
    return dict(op=op, nx=nx, ny=ny, nz=nz, ncam=ncam, psf=psf, att=att, dtype=dtype, arc=arc, tilt=tilt, **more)


def listed():
    return [
        # one call on a small grid: a test, a phantom study, an interactive preview
        dict(_case("project", 32, 32, 32, 8, psf=7), name="project_32"),
        # plain MLEM iteration of the reference's small example
        dict(_case("osem", 64, 64, 64, 60, att=False, subsets=1), name="mlem_64"),
        # the drop-in calls on host arrays, as the reference's Python package makes them
        dict(_case("host", 96, 96, 80, 90, psf=11), name="host_96"),
        # half-turn acquisition on an odd grid, a reconstruction's backprojection
        dict(_case("backproject", 111, 93, 111, 72, psf=9, arc=180), name="backproject_111"),
        # the full emission model: projection and backprojection in one call
        dict(_case("pair", 128, 128, 128, 120, psf=11), name="pair_128"),
        # one OSEM iteration over interleaved subsets with a plan
        dict(_case("osem", 128, 128, 128, 120, psf=11, subsets=8), name="osem_128"),
        # projector inside a differentiable model: forward, d/d(activity), d/d(mu)
        dict(_case("grad", 128, 128, 128, 120, psf=11), name="grad_128"),
        # the reference's attenuation gradient (joint activity / mu estimation)
        dict(_case("attgrad", 128, 128, 128, 120, psf=11), name="attgrad_128"),
        # many patients at once: volumes of uneven size, angles and subsets
        dict(op="batch", volumes=8, first=0, trim=0, psf=11, name="batch_8"),
        # high-resolution emission model
        dict(_case("pair", 256, 256, 256, 180, psf=15), name="pair_256"),
        # the same model with activity and mu stored in bfloat16
        dict(_case("pair", 192, 192, 192, 120, psf=15, dtype="bf16"), name="pair_bf16_192"),
        # cameras off the gantry axis (tilted heads): projection, then backprojection
        dict(_case("two", 96, 96, 96, 30, psf=11, tilt=7.0), name="tilted_96"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["project", "backproject", "pair", "pair", "two", "host", "grad", "attgrad", "osem", "osem",
                     "batch"])
    if op == "batch":
        return dict(op="batch", volumes=rng.randint(2, 8), first=rng.randint(0, 23), trim=rng.choice([0, 1, 3]),
                    psf=rng.choice([7, 11]))
    limit = _voxel_cameras(listed()[9])
    while True:
        nx = _log_int(rng, 28, 256)
        ny = _log_int(rng, 28, 256)
        nz = nx if rng.random() < 0.6 else max(24, int(nx * rng.uniform(0.7, 1.2)))
        case = _case(op, nx, ny, nz, _log_int(rng, 8, 180), psf=rng.choice([0, 5, 7, 9, 11, 11, 13, 15]),
                     att=op in ("grad", "attgrad") or rng.random() < 0.75, arc=rng.choice([360, 360, 180]))
        if op == "two":  # the general-orientation path and the float64 run
            case["dtype"] = rng.choice(["f32", "f32", "f64"])
            case["tilt"] = rng.uniform(2.0, 20.0)
            if _voxel_cameras(case) > 96 ** 3 * 30:
                continue
        elif op in ("project", "backproject", "pair") and case["att"]:
            case["dtype"] = rng.choice(["f32", "f32", "bf16"])
        if op == "host":
            case["nz"] = min(nz, nx)
        if op in ("grad", "attgrad", "osem", "host") and _voxel_cameras(case) > 160 ** 3 * 120:
            continue
        if op == "osem":
            case["subsets"] = rng.choice([s for s in (1, 4, 8, 12) if s <= case["ncam"]])
        if _voxel_cameras(case) <= limit:
            return case


def _volumes(case):
    """The batched reconstruction's volumes: grids, angles and subsets mixed."""
    grids = [(64, 64, 64), (96, 96, 80), (128, 128, 128), (160, 160, 128)]
    angles = [60, 90, 120, 180]
    subsets = [4, 8, 12, 16]
    out = []
    for j in range(case["volumes"]):
        i = case["first"] + j
        nx, ny, nz = (n - case["trim"] for n in grids[i % 4])
        out.append(_case("osem", nx, ny, nz, angles[(i // 4 + i) % 4], psf=case["psf"], subsets=subsets[(i // 2) % 4]))
    return out


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda", 0)


def _ellipsoids(shape, specs):
    """Sum of value over ellipsoids (centre, semi-axes in voxels x, y, z; rotation)."""
    nz, ny, nx = shape
    dev = _device()
    x = torch.arange(nx, device=dev, dtype=torch.float32)[None, None, :]
    y = torch.arange(ny, device=dev, dtype=torch.float32)[None, :, None]
    z = torch.arange(nz, device=dev, dtype=torch.float32)[:, None, None]
    vol = torch.zeros(shape, device=dev)
    for centre, semi, rot, value in specs:
        d = (x - centre[0], y - centre[1], z - centre[2])
        q = sum(((d[0] * rot[0][k] + d[1] * rot[1][k] + d[2] * rot[2][k]) / semi[k]) ** 2 for k in range(3))
        vol = vol + value * (q <= 1.0)
    return vol


def _rotation(rng):
    a, b, c, d = rng.normal(size=4)
    n = math.sqrt(a * a + b * b + c * c + d * d)
    a, b, c, d = a / n, b / n, c / n, d / n
    return [[a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c)],
            [2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b)],
            [2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d]]


_EYE = [[1.0, 0.0, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]]


def _activity(shape, seed):
    rng = np.random.default_rng([seed, 1])
    dims = np.array(shape[::-1], dtype=np.float64)
    specs = [((dims - 1) / 2, 0.45 * dims, _EYE, 0.1)]
    for _ in range(6):
        specs.append((rng.uniform(0.3, 0.7, 3) * dims, rng.uniform(0.08, 0.25, 3) * dims, _rotation(rng),
                      float(rng.uniform(0.5, 2.0))))
    return _ellipsoids(shape, [([float(v) for v in c], [float(v) for v in s], r, v) for c, s, r, v in specs])


def _mu(shape, seed):
    rng = np.random.default_rng([seed, 2])
    dims = np.array(shape[::-1], dtype=np.float64)
    body = _ellipsoids(shape, [((dims - 1) / 2, 0.45 * dims, _EYE, 1.0)])
    mu = 0.015 * body
    for value in (0.03, 0.005):
        c = (dims - 1) / 2 + rng.uniform(-0.15, 0.15, 3) * dims
        inside = _ellipsoids(shape, [(c, rng.uniform(0.08, 0.15, 3) * dims, _rotation(rng), 1.0)]) * body
        mu = torch.where(inside > 0, torch.full_like(mu, value), mu)
    return mu


def _psf(case, seed):
    """Depth-dependent Gaussian PSF (planes, k, k), each plane summing to one;
    the host entry points want as many planes as the volume is wide."""
    k, planes = case["psf"], max(case["nx"], case["nz"])
    if k == 0:
        return None
    rng = np.random.default_rng([seed, 3])
    s = 0.5 + (0.012 + 0.008 * rng.random()) * np.arange(planes)
    u = np.arange(k) - (k - 1) / 2
    g = np.exp(-0.5 * (u[None, :] / s[:, None]) ** 2)
    p = g[:, :, None] * g[:, None, :]
    return (p / p.sum(axis=(1, 2), keepdims=True)).astype(np.float32)


def _cameras(case, seed):
    """[3, n] angles in radians, axis-major; the first angle depends on the seed."""
    n = case["ncam"]
    rng = np.random.default_rng([seed, 4])
    cams = np.zeros((3, n))
    cams[1] = np.deg2rad(rng.uniform(0.0, 10.0) + case["arc"] / n * np.arange(n))
    if case["tilt"]:
        cams[0] = np.deg2rad(case["tilt"] * np.cos(np.arange(n)))
        cams[2] = np.deg2rad(0.5 * case["tilt"] * np.sin(np.arange(n)))
    return cams.astype(np.float32)


def _generator(seed, k):
    return torch.Generator(device=_device()).manual_seed(1000 * (seed % 1000003) + k)


def _counts(case, act, cams, seed):
    """Poisson counts (n, ny, nx) of the plain (no PSF, no attenuation) projection."""
    v = act.float().permute(0, 2, 1).contiguous()
    lam = torch.stack([_sample(v, m[0]).sum(0) for m in _matrices(case, cams, torch.float32)])
    return torch.poisson(lam.clamp_min(0) * 5.0, generator=_generator(seed, 5)).permute(0, 2, 1).contiguous()


def _inputs(case, seed):
    shape = (case["nz"], case["ny"], case["nx"])
    dtype = DTYPES[case["dtype"]]
    d = {"case": case, "cams": _cameras(case, seed), "psf": _psf(case, seed)}
    d["act"] = _activity(shape, seed).to(dtype)
    d["mu"] = _mu(shape, seed).to(dtype) if case["att"] else None
    if case["op"] in ("backproject", "attgrad", "osem"):
        d["counts"] = _counts(case, d["act"], d["cams"], seed)
    if case["op"] == "osem":
        d["start"] = torch.ones(shape, device=_device())
    if case["op"] == "grad":
        d["weight"] = torch.randn((case["ncam"], case["ny"], case["nx"]), device=_device(),
                                  generator=_generator(seed, 6))
    return d


def _plan(d):
    c = d["case"]
    return Plan((c["nz"], c["ny"], c["nx"]), d["cams"], d["psf"], d["mu"], subsets=c["subsets"])


def prepare(case, seed):
    if case["op"] == "batch":
        vols = [_inputs(c, seed + 17 * i) for i, c in enumerate(_volumes(case))]
        return {"case": case, "batch": Batch([_plan(d) for d in vols]), "counts": [d["counts"] for d in vols],
                "starts": [d["start"] for d in vols]}
    d = _inputs(case, seed)
    if case["op"] == "osem":
        d["plan"] = _plan(d)
    if case["op"] == "host":
        d["act"] = d["act"].cpu().numpy()
        d["mu"] = None if d["mu"] is None else d["mu"].cpu().numpy()
    if case["op"] == "grad":
        d["act"].requires_grad_(True)
        d["mu"].requires_grad_(True)
    return d


# --------------------------------------------------------------------- run
def _pointer(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _call_parts(d):
    """The C-ABI's grid, camera and PSF arguments and the current stream."""
    c = d["case"]
    size = (ctypes.c_int * 3)(c["nx"], c["ny"], c["nz"])
    cams = d["cams"]
    csize = (ctypes.c_int * 2)(cams.shape[1], cams.shape[0])
    psf = d["psf"]
    psize = (ctypes.c_int * 3)(*(psf.shape[::-1] if psf is not None else (0, 0, 0)))
    vp = ctypes.c_void_p
    return (size, cams.ctypes.data_as(vp), csize, psf.ctypes.data_as(vp) if psf is not None else None, psize,
            vp(torch.cuda.current_stream().cuda_stream))


def _pair(d):
    c = d["case"]
    lib = _lib.load()
    size, cams, csize, psf, psize, stream = _call_parts(d)
    sino = torch.empty((c["ncam"], c["ny"], c["nx"]), device=d["act"].device)
    back = torch.empty((c["nz"], c["ny"], c["nx"]), device=d["act"].device)
    fn = lib.nrgb_project_backproject_device_bf16 if c["dtype"] == "bf16" else lib.nrgb_project_backproject_device
    st = fn(_pointer(d["act"]), _pointer(d["mu"]), size, _pointer(sino), None, _pointer(back), cams, csize, psf,
            psize, 0.0, 0.0, 1, 0, stream)
    if st:
        raise RuntimeError(f"project_backproject returned {st}")
    return sino, back


def _attgrad(d):
    size, cams, csize, psf, psize, stream = _call_parts(d)
    out = torch.empty_like(d["act"])
    st = _lib.load().nrgb_gradient_attenuation_device(
        _pointer(d["counts"]), _pointer(d["act"]), _pointer(d["mu"]), size, _pointer(out), cams, csize, psf, psize,
        0.0, 0.0, 0, stream)
    if st:
        raise RuntimeError(f"gradient_attenuation returned {st}")
    return out


def run(state):
    op = state["case"]["op"]
    if op == "batch":
        return state["batch"].osem(state["counts"], 1, activities=state["starts"])
    act, mu, cams, psf = state["act"], state["mu"], state["cams"], state["psf"]
    if op == "project":
        return precision.project(act, mu, cams, psf, truncate=True)
    if op == "backproject":
        return precision.backproject(state["counts"], mu, cams, psf, nz=state["case"]["nz"], truncate=True)
    if op == "two":
        sino = precision.project(act, mu, cams, psf, truncate=True)
        return sino, precision.backproject(sino, mu, cams, psf, nz=state["case"]["nz"], truncate=True)
    if op == "pair":
        return _pair(state)
    if op == "host":
        sino = array_api.project(act, cams, psf, mu)
        return sino, array_api.backproject(sino, cams, psf, mu, nz=state["case"]["nz"])
    if op == "grad":
        sino = autograd.project(act, mu, cams, psf)
        g_act, g_mu = torch.autograd.grad(sino, (act, mu), grad_outputs=state["weight"])
        return sino.detach(), g_act, g_mu
    if op == "attgrad":
        return _attgrad(state)
    return state["plan"].osem(state["counts"], 1, activity=state["start"])


# -------------------------------------------------------------------- work
def _voxel_cameras(case):
    return case["nx"] * case["ny"] * case["nz"] * case["ncam"]


def work(case):
    """Bytes: every input read once, every output written once.  Flops per
    voxel and camera: trilinear (bilinear on the gantry) samples, two PSF
    passes, the depth sums with one exponential."""
    if case["op"] == "batch":
        parts = [work(c) for c in _volumes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    op = case["op"]
    vol = case["nx"] * case["ny"] * case["nz"]
    sino = case["nx"] * case["ny"] * case["ncam"]
    item = {"f32": 4, "bf16": 2, "f64": 8}[case["dtype"]]
    out = 8 if case["dtype"] == "f64" else 4
    nmu = 1 if case["att"] else 0
    tri = 21 if case["tilt"] else 7
    psf = 4 * case["psf"]
    project = tri * (1 + nmu) + psf + 2 + 3 * nmu
    back = tri * (1 + nmu) + psf + 1 + 3 * nmu
    table = {  # volumes in (storage type), volumes out, sinograms in + out, flops
        "project": (1 + nmu, 0, 1, project),
        "backproject": (nmu, 1, 1, back),
        "pair": (1 + nmu, 1, 1, project + back),
        "two": (1 + nmu, 1, 1, project + back),
        "host": (1 + nmu, 1, 1, project + back),
        "grad": (2, 2, 2, 3 * project),
        "attgrad": (2, 1, 1, project + tri),
        "osem": (1 + nmu, 1, 1, project + back),
    }
    vin, vout, sinos, flops = table[op]
    return {"bytes": vol * (vin * item + vout * out) + sino * sinos * out + 4 * case["psf"] ** 2 * case["nz"],
            "flops": flops * vol * case["ncam"]}


# ------------------------------------------------------------------- exact
# The model in 64 bits with plain torch, on volumes laid out [z][x][y].
def _rotation_matrix(angles, centre, order):
    (sx, sy, sz), (cx, cy, cz) = [math.sin(a) for a in angles], [math.cos(a) for a in angles]
    r = {"x": np.array([[1, 0, 0], [0, cx, -sx], [0, sx, cx]]),
         "y": np.array([[cy, 0, sy], [0, 1, 0], [-sy, 0, cy]]),
         "z": np.array([[cz, -sz, 0], [sz, cz, 0], [0, 0, 1]])}
    m = r[order[2]] @ r[order[1]] @ r[order[0]]
    c = np.array(centre)
    return np.concatenate([m, (c - m @ c)[:, None]], axis=1)


def _matrices(case, cams, dtype=torch.float64, back=False):
    """Per camera the sampling matrices of the rotation and of its inverse;
    the reference centres a backprojection's cameras at (nx - 1) / 2 in z."""
    nz = case["nx"] if back else case["nz"]
    centre = [(case["nx"] - 1) / 2, (case["ny"] - 1) / 2, (nz - 1) / 2]
    out = []
    for a in cams.astype(np.float64).T:
        out.append((_rotation_matrix(a, centre, "xyz"), _rotation_matrix(-a, centre, "zyx")))
    return out


def _sample(vol, m):
    """Trilinear samples of vol [z][x][y] at m (x, y, z, 1), zero outside."""
    nz, nx, ny = vol.shape
    dev, dt = vol.device, vol.dtype
    x = torch.arange(nx, device=dev, dtype=dt)[None, :, None]
    y = torch.arange(ny, device=dev, dtype=dt)[None, None, :]
    z = torch.arange(nz, device=dev, dtype=dt)[:, None, None]
    rows = m[0][1] == 0 and m[2][1] == 0 and m[1][1] == 1 and m[1][0] == 0 and m[1][2] == 0  # y kept
    if rows:
        pos = [m[i][0] * x + m[i][2] * z + m[i][3] for i in (0, 2)]
        sizes, src = (nx, nz), vol.reshape(nz * nx, ny)
    else:
        pos = [m[i][0] * x + m[i][1] * y + m[i][2] * z + m[i][3] for i in (0, 2, 1)]
        sizes, src = (nx, nz, ny), vol.reshape(-1)
    low = [torch.floor(p) for p in pos]
    rel = [p - f for p, f in zip(pos, low)]
    low = [f.long() for f in low]
    out = None
    for corner in range(2 ** len(pos)):
        w, idx, ok = None, [], None
        for i, n in enumerate(sizes):
            b = (corner >> i) & 1
            k = low[i] + b
            wi = rel[i] if b else 1 - rel[i]
            inside = (k >= 0) & (k < n)
            w = wi if w is None else w * wi
            ok = inside if ok is None else ok & inside
            idx.append(k.clamp(0, n - 1))
        flat = idx[1] * nx + idx[0]
        if not rows:
            flat = flat * ny + idx[2]
        v = src.index_select(0, flat.reshape(-1)).reshape(vol.shape)
        term = v * torch.where(ok, w, torch.zeros_like(w))
        out = term if out is None else out + term
    return out


def _separated(psf, nz, dev):
    if psf is None:
        return None
    p = torch.from_numpy(psf[:nz].astype(np.float64)).to(dev)
    r = (p.shape[1] - 1) // 2
    return p[:, r, :], p[:, :, r] / p[:, r, r][:, None]


def _convolve(vol, sep):
    """Per-plane separable convolution: rows along x, then columns along y."""
    if sep is None:
        return vol
    r = (sep[0].shape[1] - 1) // 2
    for dim, kern in ((1, sep[0]), (2, sep[1])):
        n = vol.shape[dim]
        pad = [0, 0, r, r] if dim == 1 else [r, r]
        src = torch.nn.functional.pad(vol, pad)
        vol = sum(src.narrow(dim, r + k, n) * kern[:, r - k][:, None, None] for k in range(-r, r + 1))
    return vol


def _project_one(act, mu, m, sep):
    v = _convolve(_sample(act, m), sep)
    return v.sum(0) if mu is None else (v * torch.exp(-torch.cumsum(_sample(mu, m), 0))).sum(0)


def _project(act, mu, mats, sep, clamp):
    p = torch.stack([_project_one(act, mu, m[0], sep) for m in mats])
    return p.clamp_min(0) if clamp else p


def _backproject(sino, mu, mats, sep, nz, clamp=True):
    out = 0
    for s, (fwd, bwd) in zip(sino, mats):
        v = s.expand(nz, *s.shape)
        if mu is not None:
            v = v * torch.exp(-torch.cumsum(_sample(mu, fwd), 0))
        out = out + _sample(_convolve(v, sep), bwd)
    return out.clamp_min(0) if clamp else out


def _to(t):
    return None if t is None else t.detach().double().permute(0, 2, 1).contiguous()


def _from(t):
    return t.permute(0, 2, 1).contiguous()


def _exact_osem(case, d):
    act, mu, y = _to(d["start"]), _to(d["mu"]), _to(d["counts"])
    sep = _separated(d["psf"], case["nz"], act.device)
    fwd, back = _matrices(case, d["cams"]), _matrices(case, d["cams"], back=True)
    for s in range(case["subsets"]):
        idx = list(range(s, case["ncam"], case["subsets"]))
        bm = [back[i] for i in idx]
        p = _project(act, mu, [fwd[i] for i in idx], sep, True)
        ratio = y[idx] / torch.where(p < EPSILON, torch.full_like(p, EPSILON), p)
        sens = _backproject(torch.ones_like(ratio), mu, bm, sep, case["nz"])
        act = act * _backproject(ratio, mu, bm, sep, case["nz"]) / sens.clamp_min(EPSILON)
    return _from(act)


def _exact_grad(case, d):
    act, mu = _to(d["act"]).requires_grad_(True), _to(d["mu"]).requires_grad_(True)
    sep = _separated(d["psf"], case["nz"], act.device)
    weight = _to(d["weight"])
    sino, g_act, g_mu = [], 0, 0
    for i, (fwd, _) in enumerate(_matrices(case, d["cams"])):
        p = _project_one(act, mu, fwd, sep)
        ga, gm = torch.autograd.grad(p, (act, mu), grad_outputs=weight[i])
        sino.append(p.detach())
        g_act, g_mu = g_act + ga, g_mu + gm
    return _from(torch.stack(sino)), _from(g_act), _from(g_mu)


def _exact_attgrad(case, d):
    act, mu, y = _to(d["act"]), _to(d["mu"]), _to(d["counts"])
    sep = _separated(d["psf"], case["nz"], act.device)
    out = 0
    for s, (fwd, bwd) in zip(y, _matrices(case, d["cams"])):
        e = _sample(act, fwd) * torch.exp(-torch.cumsum(_sample(mu, fwd), 0))
        out = out + _sample(_convolve(s * e.flip(0).cumsum(0).flip(0), sep), bwd)
    return _from(out)


def exact(case, seed):
    if case["op"] == "batch":
        return [_exact_osem(c, _inputs(c, seed + 17 * i)) for i, c in enumerate(_volumes(case))]
    d = _inputs(case, seed)
    op = case["op"]
    if op == "osem":
        return _exact_osem(case, d)
    if op == "grad":
        return _exact_grad(case, d)
    if op == "attgrad":
        return _exact_attgrad(case, d)
    act, mu = _to(d["act"]), _to(d["mu"])
    sep = _separated(d["psf"], case["nz"], act.device)
    nz = case["nz"]
    if op == "backproject":
        return _from(_backproject(_to(d["counts"]), mu, _matrices(case, d["cams"], back=True), sep, nz))
    sino = _project(act, mu, _matrices(case, d["cams"]), sep, True)
    if op == "project":
        return _from(sino)
    back = _from(_backproject(sino, mu, _matrices(case, d["cams"], back=True), sep, nz))
    if op == "host":
        return _from(sino).cpu().numpy(), back.cpu().numpy()
    return _from(sino), back
