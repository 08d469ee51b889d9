"""The adjoint of detectors of a few rows: warps of 1 to 16 rows, sums handed over
between rows from 8 rows and 150 000 rays on, the parts of the views in one launch
dimension or the other."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import small_geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("V", [1, 2, 3, 4, 5, 7, 8, 9, 17])
def test_few_rows_vs_oracle(cuda_ok, V, M, mode):
    d = small_geometry(n=(10, 9, 6), views=83 if V < 8 else 409, U=47, V=V, pitch=0.6, length=10.0)
    views = d["projNum"]
    gL = np.random.RandomState(V).normal(size=(views * V * 47, M)).astype(np.float32)
    with Projector(d, M, mode) as pr:
        g = pr.line_integrals_adjoint(torch.from_numpy(gL.reshape(views, V, 47, M)).cuda())
        torch.cuda.synchronize()
    ref = O.line_integrals_adjoint(d, gL, M, O.TRILINEAR if mode == "trilinear" else O.TEXEMU)
    for m in range(M):
        a = g[m].double().cpu().numpy()
        # trilinear: FP32 sums of some 1e4 terms of both signs; texture emulation: weights of
        # 1/256 steps, some of which FP32 coordinates put on the other side of a step
        assert np.max(np.abs(a - ref[m])) <= (1e-5 if mode == "trilinear" else 1e-3) * np.max(np.abs(ref[m]))
