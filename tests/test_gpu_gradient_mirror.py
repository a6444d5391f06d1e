"""The reference attenuation gradient with mirror cameras (one set of samples
for a camera and its opposite) equals the one that takes every camera from its
own matrix: two float32 evaluations of one sum whose sampling positions differ
by the rounding of the angles, hence the parity tolerance of 1e-5.  Heavy
attenuation (a slab's mu beyond the forward form's range), units without a
mate, groups of one unit and more, fewer planes than slabs, truncation."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from niftyrec_gb300 import synthetic as S
from niftyrec_gb300._lib import load

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shape,ncam,k,scale,group,trunc", [((32, 20, 32), 6, 7, 1.0, 0, 0),
                                                           ((128, 24, 33), 8, 5, 200.0, 0, 0),
                                                           ((24, 40, 40), 12, 11, 1.0, 2, 1),
                                                           ((20, 136, 66), 4, 15, 1.0, 3, 0),
                                                           ((24, 33, 70), 5, 0, 1.0, 0, 1),
                                                           ((9, 12, 9), 2, 3, 400.0, 1, 0),
                                                           ((16, 16, 16), 1, 5, 1.0, 1, 0)])
def test_mirror_units_match_single_cameras(shape, ncam, k, scale, group, trunc):
    L = load()
    nz, ny, nx = shape
    act = torch.from_numpy(S.ellipsoid_phantom(shape, seed=3)).cuda()
    mu = torch.from_numpy(S.mu_map(shape, seed=3)).cuda() * scale
    psf = S.gaussian_psf(k, nz) if k else None
    c = S.cameras_about_y(max(ncam - ncam % 2, 1), 11.0)
    if ncam % 2 and ncam > 1:
        c = np.concatenate([c, S.cameras_about_y(1, 201.0)], axis=1)
    c = np.ascontiguousarray(c[:, :ncam])
    y = torch.rand((ncam, ny, nx), generator=torch.Generator().manual_seed(1)).cuda() - (0.3 if trunc else 0.0)
    vp = ctypes.c_void_p

    def run():
        out = torch.full_like(act, float("nan"))
        st = L.nrgb_gradient_attenuation_device(
            vp(y.data_ptr()), vp(act.data_ptr()), vp(mu.data_ptr()), (ctypes.c_int * 3)(nx, ny, nz),
            vp(out.data_ptr()), c.ctypes.data_as(vp), (ctypes.c_int * 2)(ncam, 3),
            psf.ctypes.data_as(vp) if k else None, (ctypes.c_int * 3)(k, k, nz if k else 0), 0.0, 0.0, trunc,
            vp(torch.cuda.current_stream().cuda_stream))
        assert st == 0
        return out.cpu().numpy()

    L.nrgb_set_backproject_group(nx, ny, nz, ncam, group)
    try:
        one = run()
        L.nrgb_set_mirror_pairs(0)
        two = run()
    finally:
        L.nrgb_set_mirror_pairs(1)
        L.nrgb_set_backproject_group(nx, ny, nz, ncam, 0)
    assert np.isfinite(one).all() and (not trunc or one.min() >= 0)
    assert rel_l2(one, two) < 1e-5
