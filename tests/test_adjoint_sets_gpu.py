"""The sets of accumulators the adjoint sums into: the gradients' rounding error where
few views or unequal parts of them fill the sets, more view groups than one launch
holds, and the same in the batch."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Batch, Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry, spectral_setup

pytestmark = pytest.mark.gpu


def geometry(n, views, U, V, spacing):
    """Rays spacing voxels apart at the rotation axis."""
    nx, ny, nz = n
    return dict(pNumX=nx, pNumY=ny, pNumZ=nz, pLengthX=0.7 * nx, pLengthY=0.7 * ny, pLengthZ=0.7 * nz, projNum=views,
                dNumU=U, dNumV=V, dSize=spacing * 0.7 * 1.5, sod=1000.0, sdd=1500.0, rotatedDirection=1)


# ray spacing, views, M, signed values, 2-norm relative error of 8 separate FP32
# sums per voxel on the same inputs (measured)
ERRORS = [
    (0.35, 2, 3, False, 4.77e-8), (0.35, 2, 2, False, 4.77e-8), (0.35, 4, 3, True, 1.062e-7), (0.35, 12, 2, True, 1.559e-7),
    (0.35, 20, 3, False, 6.38e-8), (0.35, 20, 3, True, 1.944e-7), (0.7, 2, 3, False, 4.53e-8), (0.7, 12, 3, True, 1.036e-7),
    (1.0, 7, 2, True, 8.14e-8), (1.0, 32, 3, False, 4.73e-8), (1.5, 12, 2, True, 7.97e-8), (1.5, 60, 3, True, 1.139e-7),
    (2.2, 7, 3, True, 7.19e-8), (2.2, 20, 2, True, 8.14e-8),
]


@pytest.mark.parametrize("spacing,views,M,signed,bound", ERRORS)
def test_rounding_error(cuda_ok, spacing, views, M, signed, bound):
    U, V = int(48 * 1.3 / spacing), int(30 * 1.1 / spacing)
    d = geometry((48, 44, 30), views, U, V, spacing)
    rng = np.random.RandomState(5)
    gL = (rng.normal(size=(views * V * U, M)) if signed else rng.uniform(0.5, 1.5, (views * V * U, M))).astype(np.float32)
    with Projector(d, M, "trilinear") as pr:
        g = pr.line_integrals_adjoint(torch.from_numpy(gL.reshape(views, V, U, M)).cuda())
        torch.cuda.synchronize()
    ref = np.stack(O.line_integrals_adjoint(d, gL, M, O.TRILINEAR))
    err = np.linalg.norm(np.stack([x.double().cpu().numpy() for x in g]) - ref) / np.linalg.norm(ref)
    assert err <= 1.02 * bound


@pytest.mark.parametrize("M,views", [(1, 330000), (1, 330001), (3, 90002), (4, 400003)])
def test_more_view_groups_than_one_launch_holds(cuda_ok, M, views):
    """Over 65535 view groups in the parts of the views (five of pair cells, six of single
    voxels, side by side): the views around every part's and launch's ends are
    each summed once.  The others are zero, so that a voxel takes few terms."""
    parts = 5 if M <= 2 else 6
    edges = {0, views - 1}
    for part in range(parts):
        first, last = views * part // parts, views * (part + 1) // parts
        per = 65535 if M <= 2 else 65535 // parts
        for e in [first, last, *range(first + per, last, per)]:
            edges |= {e - 1, e, e + 1}
    on = np.array(sorted(e for e in edges if 0 <= e < views))
    assert len(on) < 150
    d = small_geometry(n=4, views=views, U=2, V=2, length=4.0)
    gL = np.zeros((views, 4, M), np.float32)
    gL[on] = np.random.RandomState(4).uniform(0.5, 1.5, (len(on), 4, M))
    gL = gL.reshape(views * 4, M)
    with Projector(d, M, "trilinear") as pr:
        pr.set_launch_shape(32, 1, 1, 2)
        g = pr.line_integrals_adjoint(torch.from_numpy(gL.reshape(views, 2, 2, M)).cuda())
        torch.cuda.synchronize()
    ref = O.line_integrals_adjoint(d, gL, M, O.TRILINEAR)
    for m in range(M):
        # at most 600 rays' positive terms, some 4 flushes each: n ulp / 2 of the sum at worst is 7e-5,
        # the typical sqrt(n) 1.5e-6; a ray missed or taken twice is 1e-3 of a voxel's sum and more
        assert np.max(np.abs(g[m].double().cpu().numpy() - ref[m])) <= 7e-5 * np.max(np.abs(ref[m]))


@pytest.mark.parametrize("mode", ["trilinear", "texemu", "texture"])
@pytest.mark.parametrize("views", [1, 2])  # views per work unit
def test_batch_sets(cuda_ok, mode, views):
    """Items of several parts of views, of columns taking turns, of one of each."""
    geoms = [(geometry((20, 18, 16), 23, 60, 50, 0.45), 3), (geometry((16, 20, 12), 3, 55, 40, 0.35), 4),
             (geometry((18, 18, 14), 31, 26, 22, 1.0), 1), (geometry((18, 18, 14), 1, 50, 40, 0.4), 2),
             (geometry((20, 20, 10), 1, 20, 9, 2.0), 3)]
    prs, vols, targets, outs = [], [], [], []
    for k, (d, M) in enumerate(geoms):
        S, mu, G, D = spectral_setup(d, M, 6, 5 + k)
        pr = Projector(d, M, mode)
        pr.set_spectral_tables(S, mu, G, 2, D, 1000.0)
        vols.append([torch.from_numpy(v).cuda() for v in random_volumes(d, M, 40 + k)])
        outs.append(pr.forward(vols[-1], want_L=True))
        targets.append(outs[-1]["I"] * (1 + 0.3 * torch.rand_like(outs[-1]["I"])))
        prs.append(pr)
    b = Batch(prs)
    b.set_views(1, views)
    I = [torch.empty_like(o["I"]) for o in outs]
    grads = b.forward_adjoint(vols, targets, I_out=I)["grads"]
    torch.cuda.synchronize()
    for pr, o, t, g in zip(prs, outs, targets, grads):
        ref = pr.backward(o["L"], 2 * torch.log(o["I"] / t) / o["I"])
        torch.cuda.synchronize()
        for x, y in zip(g, ref):
            # L, I and the residual's logarithm differ by roundings (1e-6 of residuals of 0.01 to 0.3)
            assert float((x - y).norm()) <= 1e-4 * float(y.norm())
    b.close()
    for pr in prs:
        pr.close()
