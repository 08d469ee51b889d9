"""The four-material march over the column copy where its layout can go wrong:
extents of one voxel and on either side of the fill's 32 x 32 tiles, views all
round both march axes, rays that miss, graze or start inside the border, partial
warps, skipping of empty bricks, the batched kernels; and an infinite voxel's
reach, which must be its own footprints only.  Against the FP64 oracle."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Batch, Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry, spectral_setup

pytestmark = pytest.mark.gpu

GEOMS = [
    dict(n=(33, 31, 32), views=9, U=37, V=19),
    dict(n=(1, 6, 34), views=8, U=21, V=41),
    dict(n=(6, 1, 33), views=8, U=21, V=41),
    dict(n=(17, 40, 1), views=7, U=19, V=9, rot=-1),
    dict(n=(12, 12, 12), views=8, U=30, V=16, pitch=4.0),
    dict(n=(8, 8, 8), views=260, U=64, V=50, length=8.0),  # one thread per ray
]


@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
@pytest.mark.parametrize("gi", range(len(GEOMS)))
def test_four_material_march_vs_oracle(cuda_ok, gi, mode):
    d = small_geometry(**GEOMS[gi])
    vols = random_volumes(d, 4, 70 + gi)
    for v in vols:
        v[: max(1, v.shape[0] // 3)] = 0.0  # bricks to skip
    S, mu, G, D = spectral_setup(d, 4, 6, 3 + gi)
    W = O.energy_weights(d, S, G, 2, D, 1000.0)
    ref = O.forward(d, vols, mu, W, O.TRILINEAR if mode == "trilinear" else O.TEXEMU)
    dev = [torch.from_numpy(v).cuda() for v in vols]
    with Projector(d, 4, mode) as pr:
        pr.set_spectral_tables(S, mu, G, 2, D, 1000.0)
        f = pr.forward(dev, want_L=True)
        b = Batch([pr])
        g = b.forward([dev])[0]
        torch.cuda.synchronize()
        b.close()
        pr.set_skip_empty(True)
        k = pr.forward(dev, want_L=True)
        torch.cuda.synchronize()
    tol = 1e-5 if mode == "trilinear" else 1e-4
    I = ref["I"]
    assert np.max(np.abs(f["I"].double().cpu().numpy().reshape(-1) - I) / np.maximum(I, 1e-30)) < tol
    Lr = ref["L"].reshape(-1)
    scale = np.maximum(np.abs(Lr), 1e-6 * max(float(np.max(np.abs(Lr))), 1e-30))
    assert np.max(np.abs(f["L"].double().cpu().numpy().reshape(-1) - Lr) / scale) < (1e-5 if mode == "trilinear" else 1e-3)
    for o in (g, k):
        assert torch.max(torch.abs(o["I"] - f["I"]) / f["I"]).item() < 2e-6


def test_infinite_voxel_stays_in_its_footprints(cuda_ok):
    # as with the layered sampler: the same rays are infinite or NaN, the others unchanged
    d = small_geometry(n=14, views=6, U=24, V=18)
    vols = [torch.from_numpy(v).cuda() for v in random_volumes(d, 4, 5)]
    vols[2][7, 6, 5] = float("inf")
    with Projector(d, 4, "trilinear") as pr:
        a = pr.line_integrals(vols)
        pr.set_sampler("layered")
        b = pr.line_integrals(vols)
        torch.cuda.synchronize()
    assert torch.equal(torch.isfinite(a), torch.isfinite(b))
    ok = torch.isfinite(b)
    assert float((a[ok] - b[ok]).abs().max()) <= 1e-5 * float(b[ok].abs().max())
