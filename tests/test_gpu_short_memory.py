"""Where the device memory does not hold the work space of a call's camera groups,
the call runs in smaller groups: with the library's arena released and the first
allocation failing (host-side injection), every call answers as before; with both
failing it returns status 4."""
import numpy as np
import pytest

from conftest import rel_l2
from niftyrec_gb300 import array_api as A
from niftyrec_gb300 import synthetic as S
from niftyrec_gb300._lib import NiftyRecError, load

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPE = (40, 36, 40)  # nz, ny, nx
NCAM = 12


def cameras(kind):
    c = S.cameras_about_y(NCAM, 5.0)
    if kind == "x":
        c[[0, 1]] = c[[1, 0]]
    if kind == "tilted":
        c[0] = 0.2
    return c


def calls(kind):
    """{name: (call, tolerance)}: sums of the same terms in other groups, d/dmu also
    with other depth slabs (the parity tests' 1e-5)."""
    from niftyrec_gb300 import precision as P
    from niftyrec_gb300.autograd import attenuation_grad_raw, backproject_raw

    act, mu = S.ellipsoid_phantom(SHAPE, seed=4), S.mu_map(SHAPE, seed=4)
    psf, c = S.gaussian_psf(5, SHAPE[2]), cameras(kind)
    y = np.random.default_rng(1).uniform(0.5, 1.5, (NCAM,) + SHAPE[1:]).astype(np.float32)
    t = [torch.from_numpy(v).cuda() for v in (act, mu, y)]
    out = {"d/dmu": (lambda: attenuation_grad_raw(t[2], t[0], t[1], c, psf).cpu().numpy(), 1e-5),
           "gradient": (lambda: A.gradient_attenuation(y, act, mu, c, psf), 1e-6)}
    if kind == "tilted":
        out["project"] = (lambda: A.project(act, c, psf, mu), 1e-6)
        out["backproject"] = (lambda: A.backproject(y, c, psf, mu, nz=SHAPE[0]), 1e-6)
        out["adjoint"] = (lambda: backproject_raw(t[2], t[1], c, psf, nz=SHAPE[0], mode=1).cpu().numpy(), 1e-6)
        out["partial"] = (lambda: A.project_partial(act, c, psf, mu)[1], 1e-6)
        out["float64"] = (lambda: P.project(t[0].double(), t[1].double(), c, psf).cpu().numpy(), 1e-12)
    return out


@pytest.mark.parametrize("kind", ["y", "x", "tilted"])
def test_smaller_groups_where_memory_is_short(kind):
    L = load()
    try:
        for name, (call, tol) in calls(kind).items():
            want = call()
            assert L.et_array_reset_gpu() == 0
            L.nrgb_debug_fail_allocations(1)
            got = call()
            assert np.isfinite(got).all() and rel_l2(got, want) < tol, name
            assert L.et_array_reset_gpu() == 0
            L.nrgb_debug_fail_allocations(2)
            with pytest.raises(NiftyRecError) as e:
                call()
            assert e.value.status == 4, name
    finally:
        L.nrgb_debug_fail_allocations(0)
