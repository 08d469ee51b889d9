"""The axis sampler with one thread per ray (plans of over 700 000 rays; smaller ones
share a ray among lanes): ragged detectors and view counts, every kind of launch
shape, skipping and the focal spot, against the FP64 oracle."""
import functools

import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry, spectral_setup

pytestmark = pytest.mark.gpu

GEOM = dict(n=(9, 8, 7), views=827, U=37, V=23)  # 703 777 rays; every extent ragged
SHAPES = [
    (16, 8, 2, 4), (16, 16, 4, 2), (32, 8, 1, 3), (8, 16, 3, 5), (64, 4, 2, 4), (8, 32, 5, 3),  # 8 rows a warp
    (8, 4, 1, 2), (16, 4, 2, 4), (24, 4, 4, 3),                                                 # 4 rows a warp
    (32, 1, 1, 2), (64, 2, 2, 4), (4, 32, 1, 3), (20, 8, 4, 2),                                 # run as 16 x 16
]


def problem():
    """Geometry, volumes, spectral tables."""
    d = small_geometry(**GEOM)
    assert d["projNum"] * d["dNumU"] * d["dNumV"] > 700000
    return d, random_volumes(d, 4, 71), spectral_setup(d, 4, 6, 72)


@functools.lru_cache(maxsize=None)
def oracle_L():
    d, vols, _ = problem()
    return O.line_integrals(d, vols, O.TRILINEAR).reshape(d["projNum"], d["dNumV"], d["dNumU"], 4)


def scaled(x, ref, floor):
    """Largest error relative to max(|ref|, floor * max|ref|)."""
    x = x.double().cpu().numpy()
    return float(np.max(np.abs(x - ref) / np.maximum(np.abs(ref), floor * np.max(np.abs(ref)))))


@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_launch_shapes(cuda_ok, M, mode):
    d, vols, (S, mu, G, D) = problem()
    dev = [torch.from_numpy(v).cuda() for v in vols[:M]]
    with Projector(d, M, mode) as pr:
        pr.set_spectral_tables(S, mu[:, :M], G, 2, D, 1000.0)
        first = pr.forward(dev, want_L=True)
        if mode == "trilinear":
            # the forward parity tests' bounds
            Lref = oracle_L()[..., :M]
            assert scaled(first["L"], Lref, 1e-6) < 1e-5
            W = np.asarray(O.energy_weights(d, S, G, 2, D, 1000.0), np.float64).reshape(len(S), -1)
            T = np.exp(-Lref.reshape(d["projNum"], -1, M) @ mu[:, :M].T.astype(np.float64))
            assert scaled(first["I"], np.einsum("pke,ek->pk", T, W).reshape(Lref.shape[:3]), 0.0) < 1e-5
        else:
            pr.set_sampler("layered")
            same = pr.forward(dev, want_L=True)
            pr.set_sampler("axis")
            for k, floor in (("L", 1e-6), ("I", 0.0), ("IAbsorb", 1e-6)):
                assert scaled(first[k], same[k].double().cpu().numpy(), floor) < 1e-6, k
        for shape in SHAPES:
            pr.set_launch_shape(*shape)
            out = pr.forward(dev, want_L=True)
            part = pr.forward(dev, want_L=True, views=(401, 13))
            torch.cuda.synchronize()
            # each ray is marched alone, so not even a rounding differs
            for k in ("L", "I", "IAbsorb"):
                assert torch.equal(out[k], first[k]), (shape, k)
                assert torch.equal(part[k], first[k][401:414]), (shape, k)


@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_skip_empty(cuda_ok, M, mode):
    d, _, _ = problem()
    d = dict(d, pNumX=36, pNumY=24, pNumZ=20)
    rng = np.random.RandomState(4)
    dev = []
    for m in range(M):
        v = np.zeros((20, 24, 36), np.float32)
        v[3:6, 2 + m:9, 20:31] = rng.uniform(0.5, 1.5, (3, 7 - m, 11))
        dev.append(torch.from_numpy(v).cuda())
    with Projector(d, M, mode) as pr:
        full = pr.line_integrals(dev)
        pr.set_skip_empty(True)
        skip = pr.line_integrals(dev)
        torch.cuda.synchronize()
    assert float(full.max()) > 0.1
    # the same non-zero terms in the same blocks
    assert scaled(skip, full.double().cpu().numpy(), 1e-6) < 1e-6


@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_focal_spot_equals_layered(cuda_ok, M):
    d, vols, _ = problem()
    rng = np.random.RandomState(9)
    fu, fv = rng.uniform(-0.6, 0.6, (2, d["projNum"])).astype(np.float32)
    dev = [torch.from_numpy(v).cuda() for v in vols[:M]]
    with Projector(d, M, "trilinear") as pr:
        pr.set_focal_spot(fu, fv)
        a = pr.line_integrals(dev)
        pr.set_sampler("layered")
        b = pr.line_integrals(dev)
        torch.cuda.synchronize()
    assert scaled(a, b.double().cpu().numpy(), 1e-6) < 1e-6
