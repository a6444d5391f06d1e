"""d/dmu with mirror cameras: a unit's two cameras share samples and scatter,
so the gradient must equal the one that takes every camera from its own matrix.
Both are float32 evaluations of one sum whose sampling positions differ by the
rounding of the angles, hence the parity tolerance of 1e-5.  Heavy attenuation
(a slab's mu beyond the forward form's range), units without a mate, several
scratch groups, row windows and both summation forms."""
import numpy as np
import pytest

from conftest import rel_l2
from niftyrec_gb300 import synthetic as S
from niftyrec_gb300._lib import load

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shape,ncam,k,scale,group", [((32, 20, 32), 6, 7, 1.0, 0), ((33, 24, 33), 8, 5, 150.0, 0),
                                                     ((24, 40, 40), 12, 11, 1.0, 2), ((20, 136, 66), 4, 15, 1.0, 3),
                                                     ((24, 33, 70), 5, 0, 1.0, 0), ((9, 12, 9), 2, 3, 400.0, 1)])
@pytest.mark.parametrize("det", [False, True])
def test_mirror_units_match_single_cameras(shape, ncam, k, scale, group, det):
    from niftyrec_gb300.autograd import attenuation_grad_raw, set_deterministic

    L = load()
    nz, ny, nx = shape
    act = torch.from_numpy(S.ellipsoid_phantom(shape, seed=3)).cuda()
    mu = torch.from_numpy(S.mu_map(shape, seed=3)).cuda() * scale
    psf = S.gaussian_psf(k, nz) if k else None
    # 2 x ncam/2 opposite cameras, for odd ncam one more without a mate
    c = S.cameras_about_y(ncam - ncam % 2, 11.0)
    if ncam % 2:
        c = np.concatenate([c, S.cameras_about_y(1, 201.0)], axis=1)
    g = torch.randn((ncam, ny, nx), generator=torch.Generator().manual_seed(1)).cuda()
    prev = set_deterministic(det)
    L.nrgb_set_backproject_group(nx, ny, nz, ncam, group)
    try:
        one = attenuation_grad_raw(g, act, mu, c, psf)
        L.nrgb_set_mirror_pairs(0)
        two = attenuation_grad_raw(g, act, mu, c, psf)
    finally:
        L.nrgb_set_mirror_pairs(1)
        L.nrgb_set_backproject_group(nx, ny, nz, ncam, 0)
        set_deterministic(prev)
    assert torch.isfinite(one).all()
    assert rel_l2(one.cpu().numpy(), two.cpu().numpy()) < 1e-5
