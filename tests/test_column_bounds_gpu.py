"""What the z-fastest copy and accumulators are addressed with: nothing but the
march's own clip keeps a footprint inside them, so it has to hold where a step
crosses the whole volume."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry

pytestmark = pytest.mark.gpu

# 4 voxels of 1e-8 mm along y: a step along y crosses 5e7 voxels, and the
# central ray of views 1 and 3 has a sample within 1e-6 of a step of the volume,
# 40 voxels outside it
FLAT = dict(pNumX=16, pNumY=4, pNumZ=16, pLengthX=15.99816608428955, pLengthY=4e-8, pLengthZ=16.0, projNum=4,
            dNumU=31, dNumV=17, dSize=1.0, sod=512.0, sdd=1024.0, rotatedDirection=1)


def test_flat_volume_samples_stay_inside(cuda_ok):
    vols = random_volumes(FLAT, 4, 3)
    gL = np.random.RandomState(1).normal(size=(4 * 17 * 31, 4)).astype(np.float32)
    with Projector(FLAT, 4, "trilinear") as pr:
        L = pr.line_integrals([torch.from_numpy(v).cuda() for v in vols])
        g = pr.line_integrals_adjoint(torch.from_numpy(gL.reshape(4, 17, 31, 4)).cuda())
        torch.cuda.synchronize()
    # y coordinates reach 5e10 voxels, so a few FP64 roundings move a sample by
    # up to 5e-5 voxel, and its value by that much of the largest
    ref = O.line_integrals(FLAT, vols, O.TRILINEAR).reshape(4, 17, 31, 4)
    assert np.max(np.abs(L.double().cpu().numpy() - ref)) <= 1e-4 * np.max(ref)
    ref = O.line_integrals_adjoint(FLAT, gL, 4, O.TRILINEAR)
    for m in range(4):
        assert np.max(np.abs(g[m].double().cpu().numpy() - ref[m])) <= 1e-4 * np.max(np.abs(ref[m]))


@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_texemu_marches_one_set_of_samples(cuda_ok, M):
    """At a source distance where FP32 coordinates are off by voxels, the clip
    in FP64 decides which samples count: the same ones in every sampler and in
    the adjoint."""
    d = small_geometry(n=(24, 22, 20), views=7, U=33, V=19, sod=2e7, sdd=3e7)
    vols = [torch.from_numpy(v).cuda() for v in random_volumes(d, M, 3)]
    gL = torch.from_numpy(np.random.RandomState(1).uniform(0.5, 1.5, (7, 19, 33, M)).astype(np.float32)).cuda()
    with Projector(d, M, "texemu") as pr:
        L = pr.line_integrals(vols)
        g = pr.line_integrals_adjoint(gL)
        pr.set_sampler("layered")
        ref = pr.line_integrals(vols)
        torch.cuda.synchronize()
    assert float(ref.max()) > 1.0
    # FP32 sums of the same terms in another order
    assert float((L - ref).abs().max()) <= 2e-6 * float(ref.max())
    # <gL, A x> = <A^T gL, x>, both sides sums of positive terms
    a = float((gL.double() * L.double()).sum())
    b = sum(float((x.double() * v.double()).sum()) for x, v in zip(g, vols))
    assert abs(a - b) <= 2e-6 * a
