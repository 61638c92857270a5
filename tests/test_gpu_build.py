"""BVH builds at the sizes where the builder changes shape (tiles of 256
clusters, the last 1024 in one block), in every layout, against the oracle."""
import numpy as np
import pytest

from rustracer_gb300 import scenes
from test_gpu_trace import assert_hits_equal, oracle_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntri", [2, 3, 255, 257, 1023, 1024, 1025, 1281, 9000])
def test_build_sizes(gpu_ctx, ntri):
    from rustracer_gb300 import gbrt
    sd = scenes.random_soup(ntri, seed=ntri, size=0.15)
    rays = scenes.random_rays(3000, seed=7)
    ref = oracle_scene(sd).trace(rays)[0]
    sc = gbrt.Scene(gpu_ctx, sd)
    for width in (8, 4, 2):
        sc.set_tuning(width)
        assert_hits_equal(sc.trace(rays)[0], ref)
    assert sc.info()["world_triangles"] == ntri


def test_build_order_of_sizes(gpu_ctx):
    """Scratch memory kept from a large build serves smaller and larger ones after it."""
    from rustracer_gb300 import gbrt
    rays = scenes.random_rays(2000, seed=8)
    for ntri in (4000, 50, 20_000, 1):
        sd = scenes.random_soup(ntri, seed=ntri, size=0.15)
        sc = gbrt.Scene(gpu_ctx, sd)
        sc.create_top_as()
        assert_hits_equal(sc.trace(rays)[0], oracle_scene(sd).trace(rays)[0])
