"""The energy weights' table: any number of energies (groups of four and a rest), on
detectors that fill its blocks of pixels and that do not, and what it takes of memory."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry, spectral_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 2, 3, 4, 5, 7, 8, 62, 256])
@pytest.mark.parametrize("U,V", [(1, 1), (5, 3), (4, 8), (33, 1), (1, 17), (37, 25)])
def test_energies_and_detectors(cuda_ok, U, V, E):
    d = small_geometry(n=12, views=5, U=U, V=V, pitch=1.1, length=12.0)
    vols = random_volumes(d, 2, 5)
    S, mu, G, D = spectral_setup(d, 2, E, 6)
    W = O.energy_weights(d, S, G, 2, D, 1000.0)
    ref = O.forward(d, vols, mu, W, O.TRILINEAR)
    dev = [torch.from_numpy(v).cuda() for v in vols]
    with Projector(d, 2, "trilinear") as pr:
        pr.set_spectral_tables(S, mu, G, 2, D, 1000.0)
        out = pr.forward(dev, want_L=True)
        again = pr.spectral_from_L(out["L"])
        torch.cuda.synchronize()
    # the forward parity tests' bounds
    for k, at in (("I", 1e-5), ("IAbsorb", 1e-5)):
        r = np.asarray(ref[k]).reshape(5, V, U)
        for o in (out, again):
            assert np.max(np.abs(o[k].double().cpu().numpy() - r) / np.maximum(np.abs(r), 1e-6 * np.max(r) + 1e-30)) < at, k
    assert np.max(np.abs(out["I0"].double().cpu().numpy().reshape(-1) / W.sum(axis=0).reshape(-1) - 1)) < 1e-6


def test_one_energy_takes_no_padding(cuda_ok):
    """4096 x 4096 pixels, one energy: W and I0, 64 MB each (and what the allocator
    rounds up to)."""
    d = small_geometry(n=8, views=1, U=4096, V=4096, pitch=0.01)
    with Projector(d, 1, "trilinear") as pr:
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        pr.set_spectral_tables(np.ones(1, np.float32), np.full((1, 1), 0.02, np.float32), I0Val=1000.0)
        assert free - torch.cuda.mem_get_info()[0] <= 2 * (64 << 20) + (16 << 20)
