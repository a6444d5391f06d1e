"""General-orientation path in groups of cameras: sizes around the tiles (32 x 32
of the convolution, 32 x 8 of the resampling, 8 depth planes of the scans),
camera counts below, at and above a group of 8, PSF radii with and without the
fused convolution, against the oracle (1e-5 as in the parity tests; float64
1e-12)."""
import numpy as np
import pytest

from conftest import rel_l2
from niftyrec_gb300 import array_api as A
from niftyrec_gb300 import synthetic as S
from oracle.oracle import Restated

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cameras(n, seed=0):
    rng = np.random.default_rng(seed)
    c = S.cameras_about_y(n, 5.0)
    c[0] = rng.uniform(-0.3, 0.3, n)
    c[2] = rng.uniform(-0.3, 0.3, n)
    return c.astype(np.float32)


@pytest.mark.parametrize("shape,n,k,bg", [((33, 33, 33), 8, 1, 0.0), ((31, 9, 32), 9, 3, 0.3), ((8, 40, 65), 17, 5, 0.0),
                                          ((7, 31, 34), 1, 7, 0.2), ((17, 64, 32), 3, 9, 0.0), ((9, 1, 40), 7, 0, 0.0),
                                          ((12, 35, 36), 10, 11, 0.4), ((16, 33, 30), 2, 13, 0.0),
                                          ((20, 20, 22), 8, 15, 0.0), ((20, 22, 36), 9, 17, 0.1)])
def test_general_groups(shape, n, k, bg):
    from niftyrec_gb300 import precision as P
    from niftyrec_gb300.autograd import backproject_raw

    nz, ny, nx = shape
    act, mu = S.ellipsoid_phantom(shape, seed=8), S.mu_map(shape, seed=8)
    psf = S.gaussian_psf(k, nx, 0.5, 0.03) if k else None
    c = cameras(n)
    o = Restated("f32")
    so = o.project(act, c, psf, mu, bg, 0.01 * bg)
    s = A.project(act, c, psf, mu, bg, 0.01 * bg)
    assert A.last_path() == 2
    assert max(rel_l2(s[i], so[i]) for i in range(n)) < 1e-5
    assert rel_l2(A.project(act, c, psf), o.project(act, c, psf)) < 1e-5
    bo = o.backproject(so, c, psf, mu, bg, 0.01 * bg, nz=nz)
    assert rel_l2(A.backproject(so, c, psf, mu, bg, 0.01 * bg, nz=nz), bo) < 1e-5
    go = o.gradient_attenuation(so, act, mu, c, psf, bg, 0.01 * bg)
    assert rel_l2(A.gradient_attenuation(so, act, mu, c, psf, bg, 0.01 * bg), go) < 1e-5
    for rotate in (0, 1):
        ps, pp = A.project_partial(act, c, psf, mu, bg, rotate_partial=rotate)
        pso, ppo = o.project_partial(act, c, psf, mu, bg, rotate=rotate)
        assert rel_l2(ps, pso) < 1e-5 and rel_l2(pp, ppo) < 1e-5
    t = [torch.from_numpy(x.astype(np.float64)).cuda() for x in (so, act, mu)]
    at = backproject_raw(t[0].float(), t[2].float(), c, psf, nz=nz, mode=1)
    assert rel_l2(at.cpu().numpy(), o.backproject(so, c, psf, mu, truncate=0, adjoint=True, nz=nz)) < 1e-5
    o64 = Restated("f64")
    s64 = o64.project(act, c, psf, mu)
    assert rel_l2(P.project(t[1], t[2], c, psf, truncate=True).cpu().numpy(), s64) < 1e-12
    b64 = P.backproject(torch.from_numpy(s64).cuda(), t[2], c, psf, nz=nz, truncate=True)
    assert rel_l2(b64.cpu().numpy(), o64.backproject(s64, c, psf, mu, nz=nz)) < 1e-12


def test_psf_with_a_coefficient_that_is_not_finite():
    """Taps outside the plane are skipped, not multiplied by zero."""
    shape = (10, 20, 24)
    act = S.ellipsoid_phantom(shape, seed=8)
    psf = S.gaussian_psf(5, 24)
    psf[:, 2, 4] = np.inf  # the last row tap
    s = A.project(act, cameras(2), psf)
    so = Restated("f32").project(act, cameras(2), psf)
    assert np.array_equal(np.isfinite(s), np.isfinite(so))
    ok = np.isfinite(so)
    assert ok.any() and not ok.all()
    assert rel_l2(s[ok], so[ok]) < 1e-5
