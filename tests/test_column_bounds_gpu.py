"""What the z-fastest copy and accumulators are addressed with: nothing but the
march's own clip keeps a footprint inside them, so it has to hold where a step
crosses the whole volume."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import random_volumes

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
