"""How accurately a ray is summed.  Rays shared by lanes against rays of one thread:
the same rays through a plan small enough to share them and through one of 64 or
16 times the views, both against the FP64 oracle."""
import numpy as np
import pytest
import torch

from ct_forward_projection_b200 import Projector
from oracle import oracle as O
from tests.conftest import random_volumes, small_geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [2, 4])
@pytest.mark.parametrize("views,more", [(4, 64), (16, 16)])  # 16 384 rays: 8 lanes; 65 536: 4 lanes
def test_split_sums_as_accurate_as_one_thread(cuda_ok, views, more, M):
    d = small_geometry(n=(128, 128, 96), views=views, U=64, V=64, length=128.0, pitch=3.0)
    vols = random_volumes(d, M, 11)
    dev = [torch.from_numpy(v).cuda() for v in vols]
    got = []
    for k in (1, more):  # a power of two: view p is view k p there, at the same FP32 angle
        with Projector(dict(d, projNum=views * k), M, "trilinear") as pr:
            got.append(pr.line_integrals(dev)[::k].double().cpu().numpy())
    ref = O.line_integrals(d, vols, O.TRILINEAR).reshape(got[0].shape)
    on = ref > 0.1 * ref.max()
    rms = [float(np.sqrt(np.mean(((g - ref)[on] / ref[on]) ** 2))) for g in got]
    assert on.sum() > 10000
    # either is an estimate from over 10 000 rays, good to about a percent
    assert rms[0] <= 1.05 * rms[1], rms


@pytest.mark.parametrize("mode", ["trilinear", "texemu"])
@pytest.mark.parametrize("views", [4, 64])  # 8 lanes a ray; 4 lanes
def test_four_materials_as_accurate_as_two(cuda_ok, views, mode):
    """The column copy's march of four materials against the texture gathers'
    march of the first two: the same samples, so the same rounding error (texture
    emulation: against the layered sampler, which compensates every sample)."""
    d = small_geometry(n=(128, 128, 96), views=views, U=64, V=64, length=128.0, pitch=3.0)
    vols = random_volumes(d, 4, 12)
    dev = [torch.from_numpy(v).cuda() for v in vols]
    got = {}
    for M in (2, 4):
        with Projector(d, M, mode) as pr:
            got[M] = pr.line_integrals(dev[:M])[..., :2].double().cpu().numpy()
            if mode == "texemu" and M == 2:
                pr.set_sampler("layered")
                ref = pr.line_integrals(dev[:M]).double().cpu().numpy()
    if mode == "trilinear":
        ref = O.line_integrals(d, vols[:2], O.TRILINEAR).reshape(got[2].shape)
    on = ref > 0.1 * ref.max()
    assert on.sum() > 10000
    rms = {M: float(np.sqrt(np.mean(((g - ref)[on] / ref[on]) ** 2))) for M, g in got.items()}
    assert rms[4] <= 1.05 * rms[2], rms
