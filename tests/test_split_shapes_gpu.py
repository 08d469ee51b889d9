"""Rays shared by lanes: detectors of fewer rows than a warp covers, and plans on
either side of the numbers of rays at which the lanes per ray change."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry, spectral_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("U,V,views", [(41, 1, 9), (41, 1, 700), (13, 2, 11), (13, 2, 2000), (7, 3, 5), (30, 3, 900), (5, 5, 4000)])
def test_few_rows_vs_oracle(cuda_ok, U, V, views, M):
    d = small_geometry(n=(12, 11, 9), views=views, U=U, V=V, pitch=0.8, length=12.0)
    vols = random_volumes(d, M, 8)
    S, mu, G, D = spectral_setup(d, M, 7, 4)
    W = O.energy_weights(d, S, G, 2, D, 1000.0)
    ref = O.forward(d, vols, mu, W, O.TRILINEAR)
    with Projector(d, M, "trilinear") as pr:
        pr.set_spectral_tables(S, mu, G, 2, D, 1000.0)
        out = pr.forward([torch.from_numpy(v).cuda() for v in vols], want_L=True)
        torch.cuda.synchronize()
    # the forward parity tests' bounds
    for k in ("I", "IAbsorb", "L"):
        r = np.asarray(ref[k], np.float64).reshape(out[k].shape)
        assert np.max(np.abs(out[k].double().cpu().numpy() - r) / np.maximum(np.abs(r), 1e-6 * np.max(np.abs(r)))) < 1e-5, k


@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
@pytest.mark.parametrize("skip", [False, True])
@pytest.mark.parametrize("M", [2, 4])
@pytest.mark.parametrize("U,V,views", [
    (37, 16, 24), (37, 16, 25),                      # 14 208 rays: the last of 8 lanes, 4 materials
    (37, 16, 32), (37, 16, 33),                      # 18 944: fewer materials
    (37, 32, 24), (37, 32, 25), (37, 32, 32), (37, 32, 33),  # 28 416, 37 888: of 4 lanes
    (40, 25, 350), (40, 25, 372),                    # 2 lanes; over 5 500 rays a voxel of nx + ny where empty space is skipped
    (40, 25, 700), (40, 25, 701),                    # the last of 2 lanes; one thread per ray
])
def test_equals_layered(cuda_ok, U, V, views, M, skip, mode):
    d = small_geometry(n=(64, 70, 6), views=views, U=U, V=V, pitch=2.9, length=70.0)
    vols = random_volumes(d, M, 3)
    for v in vols:
        v[:, :33] = 0.0  # bricks to skip
    dev = [torch.from_numpy(v).cuda() for v in vols]
    with Projector(d, M, mode) as pr:
        pr.set_sampler("layered")
        a = pr.line_integrals(dev)
        pr.set_sampler("axis")
        pr.set_skip_empty(skip)
        b = pr.line_integrals(dev)
        S, mu, G, D = spectral_setup(d, M, 3, 4, grid=False, det=False)
        pr.set_spectral_tables(S, mu, None, 0, None, 1000.0)
        part = pr.forward(dev, want_L=True, views=(views // 3, 7))["L"]
        torch.cuda.synchronize()
    top = float(a.abs().max())
    # the same samples and weights, summed in another order
    assert float(((a - b).abs() / a.abs().clamp_min(1e-3 * top)).max()) < 2e-6
    # a range of the views sums a ray as the whole call does
    assert torch.equal(part, b[views // 3: views // 3 + 7])
