"""The adjoint's z-fastest accumulators at the sizes where their layout, the
32 x 32 fold tiles and the warp's row groups can go wrong: one voxel or one
detector pixel along an axis, extents on either side of a tile, detectors whose
rows leave partial warps and whose rays lie closer than a voxel, every material
count (pair cells up to two, merged single voxels above) and several launch
shapes, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import small_geometry

pytestmark = pytest.mark.gpu

# relative to the largest gradient value: an FP32 sum of n terms in any order is
# within n ulp of the sum of their magnitudes; the largest voxels here collect
# under 2000 weights, and rounding grows like the square root in practice
TOL = 1e-5

GEOMS = [
    dict(n=(33, 31, 32), views=4, U=37, V=19),
    dict(n=(5, 40, 1), views=3, U=9, V=7),
    dict(n=(1, 6, 34), views=3, U=5, V=41),
    dict(n=(16, 16, 16), views=3, U=1, V=33, pitch=0.7),
    dict(n=(16, 18, 65), views=2, U=20, V=1),
    dict(n=(12, 12, 12), views=3, U=23, V=50, pitch=0.4, rot=-1),
]


@pytest.mark.parametrize("shape", [None, (4, 8, 1, 2), (64, 4, 3, 2)])
@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("gi", range(len(GEOMS)))
def test_adjoint_accumulators_vs_oracle(cuda_ok, gi, M, mode, shape):
    if shape is not None and (mode == "texemu" or gi not in (0, 5)):
        pytest.skip("launch shapes are covered on two geometries")
    d = small_geometry(**GEOMS[gi])
    rng = np.random.RandomState(60 + gi)
    n = d["projNum"] * d["dNumV"] * d["dNumU"]
    gL = rng.normal(size=(n, M)).astype(np.float32)
    gL[rng.uniform(size=n) < 0.2] = 0.0  # rays with nothing to scatter beside rays that scatter
    with Projector(d, M, mode) as pr:
        if shape is not None:
            pr.set_launch_shape(*shape)
        g = pr.line_integrals_adjoint(torch.from_numpy(gL.reshape(d["projNum"], d["dNumV"], d["dNumU"], M)).cuda())
        # a second call adds into the gradients it is given
        g2 = pr.line_integrals_adjoint(torch.from_numpy(gL.reshape(d["projNum"], d["dNumV"], d["dNumU"], M)).cuda(),
                                       grads=[x.clone() for x in g])
        torch.cuda.synchronize()
    ref = O.line_integrals_adjoint(d, gL, M, O.TRILINEAR if mode == "trilinear" else O.TEXEMU)
    # FP32 coordinates of the texture emulation flip 8-bit weights against the oracle's
    tol = TOL if mode == "trilinear" else 1e-3
    for m in range(M):
        scale = max(float(np.max(np.abs(ref[m]))), 1e-30)
        assert np.max(np.abs(g[m].double().cpu().numpy() - ref[m])) / scale < tol
        assert np.max(np.abs(g2[m].double().cpu().numpy() - 2 * ref[m])) / scale < 2 * tol
