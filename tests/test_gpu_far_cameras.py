"""Cameras whose rotation centre lies so far away that sampling positions leave
the range of a 32-bit integer: such a camera sees nothing and adds nothing, and
the other cameras of the call give what they give alone (1e-5 as in the parity
tests: other groups, depth slabs and summation orders)."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from niftyrec_gb300 import array_api as A
from niftyrec_gb300 import synthetic as S
from niftyrec_gb300._lib import load

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPE = (20, 24, 28)  # nz, ny, nx


def far_camera(axis, component, sign):
    """Half a turn about `axis` (0: x, 1: y) with a centre that puts one
    in-plane coordinate (component 0: the lateral one, 1: z) at about sign * 3e9
    while the other stays inside the grid: columns tx ty tz cx cy cz."""
    nz, ny, nx = SHAPE
    theta = np.float32(np.pi)
    s, c = float(np.sin(theta, dtype=np.float32)), float(np.cos(theta, dtype=np.float32))
    # about y: x' = cx - (cos cx + sin cz) + .., z' = cz - (-sin cx + cos cz) + ..; about x: y, z with -sin
    if axis == 0:
        s = -s
    far, span = sign * 1.5e9, (nz if component == 0 else (nx if axis == 1 else ny)) - 1
    near = (span - s * far) / (1 - c) if component == 0 else (span + s * far) / (1 - c)
    lateral, z = (far, near) if component == 0 else (near, far)
    cam = np.zeros(6)
    cam[axis], cam[5] = theta, z
    cam[3 if axis == 1 else 4] = lateral
    return cam


def near_cameras(axis, tilt):
    nz, ny, nx = SHAPE
    c = np.zeros((6, 4))
    c[axis] = np.deg2rad([3.0, 93.0, 183.0, 273.0])
    c[2] = tilt
    c[3:] = np.array([[(nx - 1) / 2], [(ny - 1) / 2], [(nz - 1) / 2]])
    return c


def gradient(y, act, mu, cams, psf):
    """The reference's attenuation gradient on device tensors."""
    vp = ctypes.c_void_p
    nz, ny, nx = act.shape
    out = torch.full_like(act, float("nan"))
    assert 0 == load().nrgb_gradient_attenuation_device(
        vp(y.data_ptr()), vp(act.data_ptr()), vp(mu.data_ptr()), (ctypes.c_int * 3)(nx, ny, nz), vp(out.data_ptr()),
        cams.ctypes.data_as(vp), (ctypes.c_int * 2)(cams.shape[1], cams.shape[0]), psf.ctypes.data_as(vp),
        (ctypes.c_int * 3)(*psf.shape[::-1]), 0.0, 0.0, 0, vp(torch.cuda.current_stream().cuda_stream))
    return out


@pytest.mark.parametrize("axis,tilt,path", [(1, 0.0, 1), (0, 0.0, 1), (1, 0.2, 2)])
@pytest.mark.parametrize("component", [0, 1])
@pytest.mark.parametrize("sign", [1, -1])
def test_far_camera_adds_nothing(axis, tilt, path, component, sign):
    from niftyrec_gb300.autograd import attenuation_grad_raw, backproject_raw, project_raw, set_deterministic

    nz, ny, nx = SHAPE
    act, mu = (torch.from_numpy(f(SHAPE, seed=4)).cuda() for f in (S.ellipsoid_phantom, S.mu_map))
    psf = S.gaussian_psf(5, nz)
    near = near_cameras(axis, tilt)
    far = far_camera(axis, component, sign)[:, None]
    assert abs(far[3:]).max() > 1e9
    both = np.ascontiguousarray(np.concatenate([near[:, :2], far, near[:, 2:]], axis=1), dtype=np.float32)
    near = np.ascontiguousarray(near, dtype=np.float32)
    keep = [0, 1, 3, 4]
    s = project_raw(act, mu, both, psf)
    assert A.last_path() == path
    assert not s[2].any()
    assert rel_l2(s[keep].cpu().numpy(), project_raw(act, mu, near, psf).cpu().numpy()) < 1e-5
    y = s + torch.rand(s.shape, generator=torch.Generator().manual_seed(2)).cuda()
    operators = [lambda g, c: backproject_raw(g, mu, c, psf, nz=nz, mode=0),
                 lambda g, c: backproject_raw(g, mu, c, psf, nz=nz, mode=1),
                 lambda g, c: attenuation_grad_raw(g, act, mu, c, psf),
                 lambda g, c: gradient(g, act, mu, c, psf)]
    for det in (False, True):
        prev = set_deterministic(det)
        try:
            for f in operators:
                one, two = f(y, both), f(y[keep].contiguous(), near)
                assert torch.isfinite(one).all()
                assert rel_l2(one.cpu().numpy(), two.cpu().numpy()) < 1e-5
        finally:
            set_deterministic(prev)


@pytest.mark.parametrize("shift", [(3e9, 0, 0), (0, 3e9, 0), (0, 0, 3e9), (-3e9, 0, 0), (0, -3e9, 0), (0, 0, -3e9)])
def test_affine_beyond_the_int_range(shift):
    m = np.eye(4, dtype=np.float32)
    m[:3, 3] = shift
    assert not A.affine(S.ellipsoid_phantom(SHAPE, seed=4) + 1.0, m).any()
