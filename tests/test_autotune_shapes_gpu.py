"""What the autotuner leaves alone: the shape of a plan whose forward has none to
choose (it is the adjoint's), and cached shapes of another kernel."""
import json
import os
import subprocess
import sys

import pytest
import torch

from ct_forward_projection_b200 import Projector
from tests.conftest import small_geometry
from tests.test_autotune_gpu import ROOT, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 4, 3, 2), (64, 4, 1, 3)])
def test_shared_rays_keep_the_plans_shape(cuda_ok, shape):
    d = small_geometry(n=(38, 36, 30), views=24, U=70, V=44)
    with Projector(d, 2, "trilinear") as pr:
        vols = setup(pr, d, 2, 4)
        pr.set_launch_shape(*shape)
        for cached in (0, 1):
            r = pr.autotune(vols, n_sample_views=7 + shape[2])
            assert (r["tile_u"], r["tile_v"], r["views_per_cta"], r["min_ctas_per_sm"]) == shape
            assert r["from_cache"] == cached and r["ms"] > 0
    # a plan of the same geometry and another shape does not take the first one's
    with Projector(d, 2, "trilinear") as pr:
        vols = setup(pr, d, 2, 4)
        r = pr.autotune(vols, n_sample_views=7 + shape[2])
        assert (r["tile_u"], r["tile_v"], r["views_per_cta"], r["min_ctas_per_sm"]) == (16, 8, 2, 4)


CHILD = r'''
import json, sys
sys.path.insert(0, {root!r})
from ct_forward_projection_b200 import Projector
from tests.conftest import small_geometry
from tests.test_autotune_gpu import setup
d = small_geometry(n=8, views=180, U=66, V=60)
with Projector(d, 4, "trilinear") as pr:
    print(json.dumps(pr.autotune(setup(pr, d, 4, 2), n_sample_views=4)))
'''


def test_cached_shape_of_another_kernel(cuda_ok, tmp_path):
    """712 800 rays, four materials: an entry without the column march's mark was
    timed with the texture gathers and does not count."""
    cache = tmp_path / "tune.txt"
    env = dict(os.environ, CTFP_TUNE_CACHE=str(cache))

    def tune():
        r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], capture_output=True, text=True, env=env,
                           cwd=ROOT, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.strip().splitlines()[-1])

    assert tune()["from_cache"] == 0 and tune()["from_cache"] == 1
    key = cache.read_text().split()[0]
    cache.write_text(key.replace("|columns", "") + " 8 8 1 2 0.5\n")
    assert tune()["from_cache"] == 0
