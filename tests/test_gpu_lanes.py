"""Narrow row windows of the fused kernels: windows of up to 64 or 32 rows run
with 16 or 8 lanes per column where the volume is wide enough.  The sizes sit
at the edges of the rule (rows 28..68, columns 32..132, a short last window of a
tall volume); each operator against the oracle, 1e-5 as in the parity tests."""
import numpy as np
import pytest

from conftest import rel_l2
from niftyrec_gb300 import array_api as A
from niftyrec_gb300 import synthetic as S
from oracle.oracle import Restated

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

RTOL = 1e-5


@pytest.fixture(scope="module")
def o32():
    return Restated("f32")


@pytest.mark.parametrize("shape,k", [((20, 32, 68), 7), ((12, 30, 132), 11), ((14, 28, 130), 15), ((16, 64, 66), 0),
                                     ((15, 61, 66), 15), ((13, 33, 65), 9), ((12, 65, 70), 5), ((10, 140, 132), 11), ((9, 80, 100), 13),
                                     ((8, 192, 98), 15), ((10, 81, 100), 11), ((9, 88, 129), 9),
                                     ((9, 160, 66), 13), ((12, 31, 32), 3), ((11, 4, 129), 5)])
@pytest.mark.parametrize("cams", ["opposite", "half-turn"])
def test_narrow_windows(o32, shape, k, cams):
    from niftyrec_gb300.autograd import attenuation_grad_raw, backproject_raw
    from niftyrec_gb300.plan import Plan

    nz, ny, nx = shape
    act, mu = S.ellipsoid_phantom(shape, seed=5), S.mu_map(shape, seed=5)
    psf = S.gaussian_psf(k, nx, 0.5, 0.04) if k else None
    c = S.cameras_about_y(4, 7.0) if cams == "opposite" else S.cameras_about_y(3, 7.0, 50.0)
    so = o32.project(act, c, psf, mu)
    s = A.project(act, c, psf, mu)
    assert A.last_path() == 1
    assert max(rel_l2(s[i], so[i]) for i in range(len(so))) < RTOL
    # rows one by one, so that a seam between windows cannot hide in the norm
    rows = np.linalg.norm(s - so, axis=(0, 2)) / np.maximum(np.linalg.norm(so, axis=(0, 2)), 1e-3)
    assert rows.max() < 1e-4
    bo = o32.backproject(so, c, psf, mu, nz=nz)
    assert rel_l2(A.backproject(so, c, psf, mu, nz=nz), bo) < RTOL
    t = [torch.from_numpy(x).cuda() for x in (so, act, mu)]
    bt = backproject_raw(t[0], t[2], c, psf, nz=nz, mode=1)
    assert rel_l2(bt.cpu().numpy(), o32.backproject(so, c, psf, mu, truncate=0, adjoint=True, nz=nz)) < RTOL
    go = o32.gradient_attenuation(so, act, mu, c, psf)
    assert rel_l2(A.gradient_attenuation(so, act, mu, c, psf), go) < RTOL
    plan = Plan(shape, c, psf, t[2])
    assert rel_l2(plan.project(t[1]).cpu().numpy(), so) < RTOL
    assert rel_l2(plan.backproject(t[0]).cpu().numpy(), bo) < RTOL
    # d/dmu: <grad, h> equals the oracle's directional difference in float64
    g = attenuation_grad_raw(t[0], t[1], t[2], c, psf).cpu().numpy().astype(np.float64)
    o64 = Restated("f64")
    h = np.random.default_rng(1).standard_normal(shape) * 1e-4
    d = o64.project(act, c, psf, mu + h, truncate=0) - o64.project(act, c, psf, mu - h, truncate=0)
    want = float(np.sum(so.astype(np.float64) * d)) / 2
    # the central difference is exact to second order in h; 1e-4 of the terms' size
    assert abs(float(np.sum(g * h)) - want) < 1e-4 * float(np.linalg.norm(g) * np.linalg.norm(h))


@pytest.mark.parametrize("shape,subsets", [((9, 12, 16), 4), ((8, 13, 15), 3), ((6, 130, 10), 5)])
def test_counts_split_in_one_launch(shape, subsets):
    """The one-launch split equals plane-by-plane selection and layout, exactly
    (16-byte and 4-byte layout kernels; a row stride that is padded)."""
    from niftyrec_gb300.plan import Plan

    nz, ny, nx = shape
    ids = np.random.default_rng(2).integers(0, subsets, 11).astype(np.int32)
    ids[:subsets] = np.arange(subsets)
    plan = Plan(shape, S.cameras_about_y(11), subsets=ids)
    y = torch.rand((11, ny, nx), device="cuda")
    parts = plan.split_counts(y)
    assert len(parts) == subsets
    for s, p in enumerate(parts):
        sel = y[torch.as_tensor(np.flatnonzero(ids == s), device="cuda")].contiguous()
        assert torch.equal(p, plan.to_column(sel))
