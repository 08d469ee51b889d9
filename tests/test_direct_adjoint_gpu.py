"""The adjoint of volumes whose z-fastest accumulators 32-bit elements do not reach,
because their border outweighs them ((nx + 4)(ny + 4)(nz + 4) of about 2^32 and
more): every sample adds into the gradients itself."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Batch, Projector

pytestmark = pytest.mark.gpu


def inner(xs, ys):
    """sum_m <x_m, y_m> in FP64, a part at a time."""
    return sum(float(torch.dot(a.double(), b.double()))
               for x, y in zip(xs, ys) for a, b in zip(x.reshape(-1).split(1 << 26), y.reshape(-1).split(1 << 26)))


def test_one_column(cuda_ok):
    """1 x 1 x 172 000 000 voxels, the rays through the middle of the column."""
    nz = 172_000_000
    d = dict(pNumX=1, pNumY=1, pNumZ=nz, pLengthX=2.0, pLengthY=2.0, pLengthZ=0.5 * nz, projNum=5, dNumU=9, dNumV=40,
             dSize=0.7, sod=300.0, sdd=450.0, rotatedDirection=1)
    v = [torch.zeros((nz, 1, 1), device="cuda") for _ in range(2)]
    for x in v:
        x[nz // 2 - 64: nz // 2 + 64] = torch.rand((128, 1, 1), device="cuda") + 0.5
    gL = torch.rand((5, 40, 9, 2), device="cuda") + 0.5
    with Projector(d, 2, "trilinear") as pr:
        L = pr.line_integrals(v)
        g = pr.line_integrals_adjoint(gL)
        torch.cuda.synchronize()
    a = float((gL.double() * L.double()).sum())
    assert a > 100.0
    # sums of positive terms in FP32, under 100 of them a voxel
    assert abs(inner(g, v) - a) <= 1e-5 * a
    del g, v, L
    torch.cuda.empty_cache()


@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
def test_one_slice(cuda_ok, mode):
    """32 768 x 26 240 x 1 voxels in the plan, and in the batch: tuned (there are no
    gradients then), then the same gradients as the plan's."""
    d = dict(pNumX=32768, pNumY=26240, pNumZ=1, pLengthX=327.68, pLengthY=262.4, pLengthZ=8.0, projNum=3, dNumU=6,
             dNumV=5, dSize=2.0, sod=1000.0, sdd=1500.0, rotatedDirection=1)
    v = torch.full((1, 26240, 32768), 0.8, device="cuda")
    v[0, ::3, ::5] = 1.3
    with Projector(d, 1, mode) as pr:
        pr.set_spectral_tables(np.full(3, 1 / 3, np.float32), np.full((3, 1), 0.02, np.float32), I0Val=1000.0)
        f = pr.forward([v], want_L=True)
        target = f["I"] * 1.25
        g = [torch.zeros_like(v)]
        b = Batch([pr])
        b.autotune([[v]], [target])
        loss = b.forward_adjoint([[v]], [target], grads=[g])["loss"]
        torch.cuda.synchronize()
        b.close()
        n = int((f["L"] > 0).sum())
        assert n > 10
        assert abs(float(loss[0]) - 90 * np.log(1.25) ** 2) < 1e-3
        gL = torch.rand_like(f["L"]) + 0.5
        a = float((gL.double() * f["L"].double()).sum())
        assert abs(inner(pr.line_integrals_adjoint(gL), [v]) - a) <= 1e-5 * a
        ref = pr.backward(f["L"], 2 * torch.log(f["I"] / target) / f["I"])
        torch.cuda.synchronize()
    worst = max(float((a - b).abs().max()) for a, b in zip(g[0].split(2048, 1), ref[0].split(2048, 1)))
    top = max(float(b.abs().max()) for b in ref[0].split(2048, 1))
    assert top > 0.0 and worst <= 1e-5 * top
    del v, g, ref
    torch.cuda.empty_cache()
