"""The batched projector on volumes wide enough for every lane count: windows of
8, 16 and 32 lanes in one launch, volumes of several windows with unequal tile
counts (a short last one, a split last one), against each plan's own OSEM with the
batch's four depth slabs and without mirror cameras: the same arithmetic per item,
1e-6 as in the other batch tests.  The launch itself: one set of row buffers for the
three lane counts, next to nothing spilled, the CTAs it is built for resident."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from niftyrec_gb300 import array_api as A
from niftyrec_gb300 import synthetic as S
from niftyrec_gb300._lib import load

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (shape (nz, ny, nx), cameras, subsets, PSF width or 0, with mu): 8 lanes; 16; 32 and 8;
# 32, 16 and 8; 32; 16 and 8 (split 80 rows); then the kernels without a PSF and without mu
VOLUMES = [((12, 30, 130), 6, 2, 11, True), ((10, 60, 66), 9, 3, 11, True), ((9, 140, 132), 8, 2, 11, True),
           ((8, 192, 98), 4, 1, 11, True), ((14, 128, 40), 6, 3, 11, True), ((9, 80, 100), 5, 1, 11, True),
           ((11, 28, 129), 6, 2, 0, True), ((9, 140, 132), 4, 2, 5, False)]


@pytest.mark.parametrize("graph", [False, True])
def test_batch_of_every_lane_count(graph):
    from niftyrec_gb300.batch import Batch
    from niftyrec_gb300.plan import Plan

    L, plans, counts = load(), [], []
    L.nrgb_set_mirror_pairs(0)
    try:
        for i, (shape, ncam, nsub, k, att) in enumerate(VOLUMES):
            nz, ny, nx = shape
            act = S.ellipsoid_phantom(shape, seed=70 + i) + np.float32(0.2)
            mu = S.mu_map(shape, seed=70 + i) if att else None
            psf = S.gaussian_psf(k, nx, 0.5, 0.04) if k else None
            # small angles: the reference's backprojector centre, (nx - 1) / 2 in z, lies outside these volumes
            cams = S.cameras_about_y(ncam, -3.0, 1.5)
            y = S.poisson_counts(A.project(act, cams, psf, mu), 60, seed=i)
            counts.append(torch.from_numpy(y).cuda())
            L.nrgb_set_project_slabs(nx, ny, nz, ncam, 4)
            plans.append(Plan(shape, cams, psf, torch.from_numpy(mu).cuda() if att else None, subsets=nsub))
    finally:
        L.nrgb_set_mirror_pairs(1)
        for (nz, ny, nx), ncam, *_ in VOLUMES:
            L.nrgb_set_project_slabs(nx, ny, nz, ncam, 0)
    ref = [p.osem(c, iterations=2, layout="column").cpu().numpy() for p, c in zip(plans, counts)]
    for i, (x, r) in enumerate(zip(Batch(plans).osem(counts, iterations=2, graph=graph), ref)):
        assert r.max() > 0.1 and rel_l2(x.cpu().numpy(), r) < 1e-6, VOLUMES[i]


@pytest.mark.parametrize("k,nz", [(0, 64), (5, 128), (7, 64), (11, 128), (15, 128), (15, 256)])
@pytest.mark.parametrize("att", [1, 0])
def test_launch_of_the_batched_projector(k, nz, att):
    out = (ctypes.c_int * 4)()
    assert load().nrgb_batch_projector_info(k, att, nz, out) == 0
    ctas, static, local, clusters = out
    row_buffers = 16 * 32 * 2 * 12  # one set for 8 lanes: 32 groups x 2 x (8 + 4 pads) chunks of 16 bytes
    assert static <= row_buffers + 64
    assert local <= 64
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # whole clusters of 4 CTAs per group of SMs: a few SMs of a group may be left over
    assert 4 * clusters > (ctas - 1) * sms and 4 * clusters >= 0.9 * ctas * sms


def test_launch_info_refuses_bad_arguments():
    out, L = (ctypes.c_int * 4)(), load()
    assert [L.nrgb_batch_projector_info(*a, out) for a in ((4, 1, 8), (17, 1, 8), (-1, 1, 8), (5, 1, 0))] == [2] * 4
