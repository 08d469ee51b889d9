"""The march of a plan of few rays, whose rays are shared by 8, 4 or 2 lanes
(chosen from the plan's rays): line integrals, intensities and absorbed
intensities on both sides of each threshold and at the remainders that matter
(rays shorter than the lanes' runs, detectors that leave rows and columns of a
warp empty, energies in every remainder of 4), against the FP64 oracle, and the
epilogue bit for bit against the one on stored line integrals."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry, spectral_setup

pytestmark = pytest.mark.gpu

# per pixel, relative to the oracle: FP32 sums of samples and energies (the
# parity bound of the forward tests)
TOL = {"trilinear": 1e-5, "texemu": 1e-4}

# rays: 8 lanes up to 20 000, 4 up to 400 000, 2 up to 700 000, then 1
CASES = [
    (dict(n=20, views=3, U=33, V=9), 4),
    (dict(n=(3, 4, 5), views=40, U=20, V=25), 5),        # 20 000: the last of 8 lanes
    (dict(n=(3, 4, 5), views=37, U=23, V=47), 6),        # 39 997: 4 lanes, rays of a few samples
    (dict(n=(5, 4, 3), views=400, U=40, V=25), 7),       # 400 000: the last of 4 lanes
    (dict(n=(5, 4, 3), views=401, U=40, V=25), 3),       # 2 lanes
    (dict(n=(5, 4, 3), views=700, U=40, V=25), 1),       # 700 000: the last of 2 lanes
    (dict(n=(5, 4, 3), views=701, U=40, V=25), 9),       # one thread per ray
    (dict(n=12, views=70000, U=1, V=1), 2),              # more views than one launch holds
]


@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
@pytest.mark.parametrize("k", range(len(CASES)))
def test_split_march_vs_oracle(cuda_ok, k, mode):
    geom, E = CASES[k]
    d = small_geometry(length=12.0, **geom)
    M = 1 + k % 4
    vols = random_volumes(d, M, 30 + k)
    S, mu, G, D = spectral_setup(d, M, E, 7 + k)
    W = O.energy_weights(d, S, G, 2, D, 1000.0)
    ref = O.forward(d, vols, mu, W, O.TRILINEAR if mode == "trilinear" else O.TEXEMU)
    with Projector(d, M, mode) as pr:
        pr.set_spectral_tables(S, mu, G, 2, D, 1000.0)
        dev = [torch.from_numpy(v).cuda() for v in vols]
        f = pr.forward(dev, want_L=True)
        s = pr.spectral_from_L(f["L"])
        L = pr.line_integrals(dev)
        torch.cuda.synchronize()
    assert torch.equal(f["L"], L)
    assert torch.equal(f["I"], s["I"]) and torch.equal(f["IAbsorb"], s["IAbsorb"])
    for key in ("I", "IAbsorb"):
        x = f[key].double().cpu().numpy().reshape(-1)
        assert np.max(np.abs(x - ref[key]) / np.maximum(np.abs(ref[key]), 1e-30)) < TOL[mode] * (10 if key == "IAbsorb" and mode == "texemu" else 1)
