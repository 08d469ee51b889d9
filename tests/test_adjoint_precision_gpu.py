"""The gradients' rounding error: no larger than that of 8 separate FP32 sums per
voxel (a face accumulator per corner and march axis), whose error on the same
inputs the bounds state; and the adjoint where memory is short."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Batch, Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry, spectral_setup

pytestmark = pytest.mark.gpu

# geometry, 2-norm relative error of 8 sums (measured, 1 to 4 materials within 1 %)
CASES = [
    (dict(n=(48, 44, 30), views=90, U=180, V=110, length=48.0, pitch=0.55), 1.30e-7),  # rays closer than a voxel
    (dict(n=(64, 60, 40), views=20, U=64, V=48, length=64.0, pitch=2.0), 4.3e-8),      # ten rays a voxel
    (dict(n=(64, 60, 40), views=4, U=100, V=70, length=64.0, pitch=1.5), 4.57e-8),     # few views
    (dict(n=(96, 96, 1), views=180, U=200, V=1, length=96.0, pitch=0.9), 1.23e-7),     # one slice, one row
]


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("k", range(len(CASES)))
def test_gradient_rounding_error(cuda_ok, k, M):
    geom, bound = CASES[k]
    d = small_geometry(**geom)
    n = d["projNum"] * d["dNumV"] * d["dNumU"]
    gL = np.random.RandomState(5).uniform(0.5, 1.5, (n, M)).astype(np.float32)
    with Projector(d, M, "trilinear") as pr:
        g = pr.line_integrals_adjoint(torch.from_numpy(gL.reshape(d["projNum"], d["dNumV"], d["dNumU"], M)).cuda())
        torch.cuda.synchronize()
    ref = np.stack(O.line_integrals_adjoint(d, gL, M, O.TRILINEAR))
    err = np.linalg.norm(np.stack([x.double().cpu().numpy() for x in g]) - ref) / np.linalg.norm(ref)
    assert err <= 1.02 * bound


def test_adjoint_with_little_memory_left(cuda_ok):
    """Five sets of accumulators (1.1 GB) do not fit into what is left: fewer
    are used, in the plan and in the batch, with the same gradients."""
    d = small_geometry(n=300, views=12, U=120, V=100, length=300.0, pitch=2.0)
    vols = [torch.from_numpy(v).cuda() for v in random_volumes(d, 1, 3)]
    S, mu, G, D = spectral_setup(d, 1, 3, 5, grid=False, det=False)
    gL = torch.rand((12, 100, 120, 1), device="cuda")
    target = torch.full((12, 100, 120), 900.0, device="cuda")

    def grads(left):
        out = []
        for use in ("plan", "batch"):
            with Projector(d, 1, "trilinear") as pr:
                pr.set_spectral_tables(S, mu, None, 0, None, 1000.0)
                g = [torch.zeros_like(vols[0])]
                torch.cuda.synchronize()
                torch.cuda.empty_cache()
                free = torch.cuda.mem_get_info()[0]
                hog = torch.empty(free - left, dtype=torch.uint8, device="cuda") if left else None
                if use == "plan":
                    pr.line_integrals_adjoint(gL, grads=g)
                else:
                    b = Batch([pr])
                    b.forward_adjoint([vols], [target], grads=[g])
                    b.close()
                torch.cuda.synchronize()
                del hog
                torch.cuda.empty_cache()
            out.append(g[0])
        return out

    for a, b in zip(grads(600 << 20), grads(0)):
        # FP32 sums of the same terms
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
