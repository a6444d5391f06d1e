"""d/dmu with a gradient pixel that is not finite: only the voxels that its ray
passes are affected, in both summation forms.  At angle 0 every sample lies on a
grid node, so a corner of weight zero must not be touched (0 * inf)."""
import numpy as np
import pytest

from niftyrec_gb300 import synthetic as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shape", [(16, 20, 16), (18, 40, 66), (12, 30, 130)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("det", [False, True])
def test_only_the_ray_is_affected(shape, value, det):
    from niftyrec_gb300.autograd import attenuation_grad_raw, set_deterministic

    nz, ny, nx = shape
    act = torch.from_numpy(S.ellipsoid_phantom(shape, seed=3)).cuda() + 0.5
    mu = torch.from_numpy(S.mu_map(shape, seed=3)).cuda() + 0.01
    cams = np.zeros((3, 2), np.float32)
    cams[1, 1] = 0.7
    g = torch.rand((2, ny, nx), generator=torch.Generator().manual_seed(1)).cuda() + 0.1
    y, x = ny // 2, nx // 2
    prev = set_deterministic(det)
    try:
        clean = attenuation_grad_raw(g, act, mu, cams)
        g[0, y, x] = value
        out = attenuation_grad_raw(g, act, mu, cams)
    finally:
        set_deterministic(prev)
    on_ray = torch.zeros(shape, dtype=torch.bool, device="cuda")
    on_ray[:, y, x] = True
    assert not torch.isfinite(out[on_ray]).any()
    assert torch.isfinite(out[~on_ray]).all()
    # float32 sums of the same terms in another order
    assert float((out - clean)[~on_ray].norm() / clean[~on_ray].norm()) < 1e-6
