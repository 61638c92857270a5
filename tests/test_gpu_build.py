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


@pytest.mark.parametrize("flags", [0, 1], ids=["flattened", "tlas"])
def test_build_many_geometries(gpu_ctx, flags):
    """Triangles of many geometries of one to forty triangles, in instances out of
    order, repeated and masked out: each hit names its instance, geometry and primitive."""
    import pyoracle as O
    from rustracer_gb300 import gbrt
    rng = np.random.default_rng(11)
    b = scenes.GeoBuilder()
    mat = b.add_material(scenes.random_pbr_material(rng))
    for n in [1, 40, 2, 1, 31, 32, 33, 7]:
        p = (rng.uniform(-1, 1, (n, 1, 3)) + rng.normal(0, 0.15, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
        b.add_mesh(p, np.arange(3 * n), mat, normal=np.tile(np.float32([0, 0, 1]), (3 * n, 1)))
    order = [7, 0, 3, 5, 1, 5, 2, 6, 4, 0]
    shift = [np.float32([1, 0, 0, x, 0, 1, 0, 0, 0, 0, 1, 0]) for x in (0, 0, .5, 0, 0, -.3, .2, 0, 0, .7)]
    sd = b.finish(instances=scenes.identity_instances(order, shift),
                  camera=dict(eye=(0, 0, 3.0), direction=(0, 0, -1), fov_deg=60.0))
    sd.instances[3]["custom_index_and_mask"] &= 0xFFFFFF
    rays = scenes.random_rays(20_000, seed=12)
    ref = O.OracleScene(sd, build_flags=flags).trace(rays)[0]
    assert len(np.unique(ref["instance_id"])) >= 8
    assert_hits_equal(gbrt.Scene(gpu_ctx, sd, build_flags=flags).trace(rays)[0], ref)


@pytest.mark.parametrize("flags", [0, 2], ids=["width8", "width4"])
def test_far_vertices(gpu_ctx, flags):
    """Two triangles so far out that the surface area of the boxes around them
    overflows: the others are found as before."""
    from rustracer_gb300 import gbrt
    sd = scenes.random_soup(2000, seed=61, size=0.15)
    sd.vertices["pos"][-6:, :3] = np.float32([[2e19, 0, 0], [2e19, 1, 0], [2e19, 0, 1], [-2e19, 2e19, -2e19],
                                              [-2e19, 2e19, -1e19], [-2e19, 1e19, -2e19]])
    rays = scenes.random_rays(5000, seed=62)
    ref = oracle_scene(sd).trace(rays)[0]
    assert (ref["instance_id"] != 0xFFFFFFFF).mean() > 0.4
    sc = gbrt.Scene(gpu_ctx, sd, build_flags=flags)
    for width in (4 if flags else 8, 2):
        sc.set_tuning(width)
        assert_hits_equal(sc.trace(rays)[0], ref)
