"""Detectors of more than 2^31 pixels a view (sides up to 65535 are accepted)."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector

pytestmark = pytest.mark.gpu


def test_spectral_from_L_past_2_31_pixels(cuda_ok):
    U, V = 65535, 32800
    assert U * V > 2 ** 31
    d = dict(pNumX=4, pNumY=4, pNumZ=4, pLengthX=4.0, pLengthY=4.0, pLengthZ=4.0, projNum=1, dNumU=U, dNumV=V,
             dSize=1e-3, sod=300.0, sdd=450.0, rotatedDirection=1)
    with Projector(d, 1, "trilinear") as pr:
        pr.set_spectral_tables(np.ones(1, np.float32), np.full((1, 1), 0.5, np.float32), I0Val=1000.0)
        L = torch.zeros((1, V, U, 1), device="cuda")
        L[0, ::97] = 1.0
        L[0, -3:] = 2.0
        r = pr.spectral_from_L(L)
        torch.cuda.synchronize()
        I = r["I"][0]
        for rows, path in ((slice(V - 3, V), 2.0), (slice(0, 97 * 300, 97), 1.0), (slice(V - 40, V - 30), None)):
            x = I[rows].double()
            want = 1000.0 * np.exp(-0.5 * path) if path is not None else \
                1000.0 * torch.exp(-0.5 * L[0, rows, :, 0].double())
            assert float(((x - want) / want).abs().max()) < 1e-6
    del L, r, I
    torch.cuda.empty_cache()
