"""Windows of 8 and 16 lanes and split last windows in the forms that
test_gpu_lanes.py does not run: bfloat16 storage, the gradients and the exact
transpose for cameras about y and about x, the deterministic forms.  The
gradients against the general path (cameras tilted by 1e-9), the whole volume to
1e-5 as in the parity tests and every row to 1e-4, so that a seam between
windows cannot hide in the norm; mirror units, a camera without a mate,
several scratch groups, truncation of signed data, heavy attenuation."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from niftyrec_gb300 import array_api as A
from niftyrec_gb300 import synthetic as S
from niftyrec_gb300._lib import load

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

RTOL = 1e-5
FUSED, GENERAL = 1, 2


def lanes(shape, k, axis=1):
    """Lanes of the row windows of a (nz, ny, nx) volume."""
    nz, ny, nx = shape
    out, n = (ctypes.c_int * 40)(), ctypes.c_int(0)
    size = (ctypes.c_int * 3)(*((nx, ny, nz) if axis == 1 else (ny, nx, nz)))
    assert load().nrgb_volume_windows(size, k, out, 8, ctypes.byref(n)) == 0
    return [out[5 * i + 4] for i in range(n.value)]


@pytest.mark.parametrize("shape,k,want", [((66, 28, 66), 11, [8]), ((66, 60, 66), 7, [16]), ((98, 80, 98), 11, [16, 8]),
                                          ((66, 140, 66), 15, [32, 8]), ((66, 30, 66), 0, [8])])
@pytest.mark.parametrize("ncam", [4, 3])
def test_bfloat16_storage(shape, k, want, ncam):
    """Mirror units (4 cameras) and single cameras (3); float64 on the same rounded
    inputs differs by float32 arithmetic only."""
    from niftyrec_gb300 import precision as P

    assert lanes(shape, k) == want
    a16 = torch.from_numpy(S.ellipsoid_phantom(shape, seed=53)).cuda().to(torch.bfloat16)
    m16 = torch.from_numpy(S.mu_map(shape, seed=53)).cuda().to(torch.bfloat16)
    psf = S.gaussian_psf(k, shape[0], 0.5, 0.03) if k else None
    cams = S.cameras_about_y(ncam, 3.0)
    p16 = P.project(a16, m16, cams, psf)
    assert A.last_path() == FUSED
    p64 = P.project(a16.double(), m16.double(), cams, psf)
    assert P.rel_error(p16, p64)[1] < RTOL
    rows = (p16.double() - p64).norm(dim=(0, 2)) / p64.norm(dim=(0, 2)).clamp_min(1e-2 * float(p64.norm(dim=(0, 2)).max()))
    assert float(rows.max()) < 1e-4
    b16 = P.backproject(p64.float(), m16, cams, psf, nz=shape[0])
    assert P.rel_error(b16, P.backproject(p64, m16.double(), cams, psf, nz=shape[0]))[0] < RTOL


def gradient(y, act, mu, cams, psf, truncate):
    """The reference's attenuation gradient on device tensors."""
    vp = ctypes.c_void_p
    nz, ny, nx = act.shape
    out = torch.full_like(act, float("nan"))
    assert 0 == load().nrgb_gradient_attenuation_device(
        vp(y.data_ptr()), vp(act.data_ptr()), vp(mu.data_ptr()), (ctypes.c_int * 3)(nx, ny, nz), vp(out.data_ptr()),
        cams.ctypes.data_as(vp), (ctypes.c_int * 2)(cams.shape[1], cams.shape[0]),
        psf.ctypes.data_as(vp) if psf is not None else None,
        (ctypes.c_int * 3)(*(psf.shape[::-1] if psf is not None else (0, 0, 0))), 0.0, 0.0, truncate,
        vp(torch.cuda.current_stream().cuda_stream))
    return out


def agree(a, b, axis):
    a, b = a.cpu().numpy(), b.cpu().numpy()
    assert np.isfinite(a).all() and rel_l2(a, b) < RTOL
    other = (0, 2) if axis == 1 else (0, 1)  # rows of the windows: y, for cameras about x nifti x
    size = np.linalg.norm(b.astype(np.float64), axis=other)
    rows = np.linalg.norm(a.astype(np.float64) - b, axis=other) / np.maximum(size, 1e-2 * size.max())
    assert rows.max() < 1e-4


CASES = [((12, 30, 130), 11, 1.0, [8]), ((10, 60, 66), 7, 1.0, [16]), ((9, 80, 100), 11, 1.0, [16, 8]),
         ((9, 140, 132), 15, 1.0, [32, 8]), ((11, 28, 129), 0, 1.0, [8]), ((40, 32, 66), 5, 100.0, [8])]


@pytest.mark.parametrize("shape,k,scale,want", CASES)
@pytest.mark.parametrize("axis", [1, 0])
@pytest.mark.parametrize("det", [False, True])
def test_gradients_against_the_general_path(shape, k, scale, want, axis, det):
    from niftyrec_gb300.autograd import attenuation_grad_raw, backproject_raw, set_deterministic

    if axis == 0:
        shape = (shape[0], shape[2], (shape[1] + 3) // 4 * 4)
    assert lanes(shape, k, axis) == want
    L, ncam = load(), 5
    nz, ny, nx = shape
    act = torch.from_numpy(S.ellipsoid_phantom(shape, seed=3)).cuda() + 0.1
    mu = torch.from_numpy(S.mu_map(shape, seed=3)).cuda() * scale
    psf = S.gaussian_psf(k, nz, 0.5, 0.03) if k else None
    cams = np.zeros((3, ncam), np.float32)
    cams[axis] = np.deg2rad([11.0, 101.0, 191.0, 281.0, 31.0])  # the last without a mate
    tilted = cams.copy()
    tilted[2] = 1e-9
    g = torch.rand((ncam, ny, nx), generator=torch.Generator().manual_seed(1)).cuda() + 0.5
    signed = g - 0.8
    calls = [(lambda c: attenuation_grad_raw(g, act, mu, c, psf)),
             (lambda c: backproject_raw(g, mu, c, psf, nz=nz, mode=1)),
             (lambda c: gradient(g, act, mu, c, psf, 0)), (lambda c: gradient(signed, act, mu, c, psf, 1))]
    prev = set_deterministic(det)
    L.nrgb_set_backproject_group(nx, ny, nz, ncam, 2)
    try:
        for i, call in enumerate(calls):
            one = call(cams)
            assert A.last_path() == FUSED
            two = call(tilted)
            assert A.last_path() == GENERAL
            agree(one, two, axis)
            if i == 3:
                assert float(one.min()) >= 0 and float(one.max()) > 0
    finally:
        L.nrgb_set_backproject_group(nx, ny, nz, ncam, 0)
        set_deterministic(prev)


@pytest.mark.parametrize("shape,k,scale,group", [((33, 24, 33), 5, 150.0, 0), ((24, 40, 40), 11, 1.0, 2),
                                                 ((20, 136, 66), 15, 1.0, 3), ((66, 30, 66), 7, 1.0, 2)])
def test_deterministic_dmu_against_mirror_units(shape, k, scale, group):
    """The deterministic form takes every camera alone; the other form shares the
    walk of two opposite cameras (rounding of the mirrored positions: 1e-5)."""
    from niftyrec_gb300.autograd import attenuation_grad_raw, set_deterministic

    L, ncam = load(), 8
    nz, ny, nx = shape
    act = torch.from_numpy(S.ellipsoid_phantom(shape, seed=3)).cuda()
    mu = torch.from_numpy(S.mu_map(shape, seed=3)).cuda() * scale
    psf, c = S.gaussian_psf(k, nz), S.cameras_about_y(ncam, 11.0)
    g = torch.rand((ncam, ny, nx), generator=torch.Generator().manual_seed(1)).cuda() + 0.5
    L.nrgb_set_backproject_group(nx, ny, nz, ncam, group)
    out = []
    try:
        for det in (True, False):
            prev = set_deterministic(det)
            out.append(attenuation_grad_raw(g, act, mu, c, psf))
            set_deterministic(prev)
    finally:
        L.nrgb_set_backproject_group(nx, ny, nz, ncam, 0)
    agree(out[0], out[1], 1)
