"""Waves and ray queries of every size class against the CPU oracle: a single
ray or path, counts around a warp and around two rays per resident warp
(152 SMs x 28 warps), where launches change shape, and images whose width and
height leave remainders in blocks and bands."""
import numpy as np
import pytest

import parity
from rustracer_gb300 import scenes, types as T
from test_gpu_render import oracle_ref, render_gpu
from test_gpu_trace import assert_hits_equal, oracle_scene

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 3, 31, 32, 33, 129, 8511, 8513, 136_197]


@pytest.fixture(scope="module")
def soup():
    sd = scenes.random_soup(3000, seed=21, size=0.1, alpha_mask_fraction=0.5)
    rays = scenes.random_rays(max(COUNTS), seed=22)
    return sd, rays, oracle_scene(sd).trace(rays)[0]


@pytest.mark.parametrize("count", COUNTS)
def test_ray_counts(gpu_ctx, soup, count):
    from rustracer_gb300 import gbrt
    sd, rays, ref = soup
    sc = gbrt.Scene(gpu_ctx, sd)
    hits, _ = sc.trace(rays[:count])
    assert_hits_equal(hits, ref[:count])
    any_hits, _ = sc.trace(rays[:count], 0x4)
    assert np.array_equal(any_hits["instance_id"] == 0xFFFFFFFF, ref[:count]["instance_id"] == 0xFFFFFFFF)


@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (1, 9, 2), (9, 1, 3), (31, 17, 1), (33, 8, 3), (8, 33, 2),
                                              (257, 65, 1)])
def test_frame_sizes(gpu_ctx, width, height, spp):
    sd = scenes.icosphere_scene(subdiv=2)
    ubo = sd.ubo(width, height, samples=spp, bounces=6, exposure=1.0)
    orc, ref = oracle_ref(sd, ubo, width, height)
    r = render_gpu(gpu_ctx, sd, ubo, width, height)
    assert_hits_equal(r["hits"].reshape(-1), ref["hits"].reshape(-1))
    c = parity.classify(r["samples"], ref, orc, ubo, width, height)
    assert c["unexplained"] == 0, c
    assert int(r["stats"]["rays_camera"]) == width * height * spp


@pytest.mark.parametrize("ntri,size,masked", [(60, 2.0, 0.0), (600, 0.8, 0.5)])
def test_crowded_leaves(gpu_ctx, ntri, size, masked):
    """Big overlapping triangles: a step of a warp turns up far more of them than it has lanes."""
    from rustracer_gb300 import gbrt
    sd = scenes.random_soup(ntri, seed=31, size=size, alpha_mask_fraction=masked)
    rays = scenes.random_rays(20_001, seed=32)
    ref = oracle_scene(sd).trace(rays)[0]
    sc = gbrt.Scene(gpu_ctx, sd)
    assert_hits_equal(sc.trace(rays)[0], ref)
    any_hits = sc.trace(rays, 0x4)[0]
    assert np.array_equal(any_hits["instance_id"] == 0xFFFFFFFF, ref["instance_id"] == 0xFFFFFFFF)


@pytest.mark.parametrize("form", ["flattened", "tlas", "binary"])
@pytest.mark.parametrize("masked", [0.0, 0.5], ids=["opaque", "masked"])
def test_ray_query_forms(gpu_ctx, form, masked):
    """Closest and any hits, with and without the alpha test, through each form of the query kernel."""
    import pyoracle as O
    from rustracer_gb300 import gbrt
    sd = scenes.random_soup(900, seed=17, extent=0.6, size=0.15, alpha_mask_fraction=masked)
    sd.instances["transform"][1] = np.float32([0.8, 0, 0, 0.3, 0, 0.8, 0, 0, 0, 0, 0.8, -0.2])
    build = gbrt.BUILD_NO_FLATTEN if form == "tlas" else 0
    sc, orc = gbrt.Scene(gpu_ctx, sd, build_flags=build), O.OracleScene(sd, build_flags=build)
    if form == "binary":
        sc.set_tuning(2)
    rays = scenes.random_rays(4097, seed=18)
    for flags in (0, 1):  # GBRT_RAY_OPAQUE
        ref = orc.trace(rays, flags)[0]
        assert_hits_equal(sc.trace(rays, flags)[0], ref)
        any_hit = sc.trace(rays, flags | 4)[0]  # GBRT_RAY_TERMINATE_ON_FIRST: some hit of the ray
        assert np.array_equal(any_hit["t"] >= 0, ref["t"] >= 0)


@pytest.mark.parametrize("per_warp", [2, 16], ids=["two rays a warp", "full warps"])
@pytest.mark.parametrize("off", [-2, -1, 0, 1])
def test_ray_counts_at_launch_shapes(gpu_ctx, soup, per_warp, off):
    """Counts where a query's launch goes from one-warp blocks to full ones (two rays
    per resident warp) and where its warps take 32 rays at a time (sixteen), of this
    GPU: eight blocks of four warps per SM."""
    import torch
    from rustracer_gb300 import gbrt
    sd, rays, ref = soup
    count = per_warp * 32 * torch.cuda.get_device_properties(0).multi_processor_count + off
    assert count < len(rays)
    sc = gbrt.Scene(gpu_ctx, sd)
    for width in (8, 2):
        sc.set_tuning(width)
        assert_hits_equal(sc.trace(rays[:count])[0], ref[:count])
        any_hits = sc.trace(rays[:count], 0x4)[0]
        assert np.array_equal(any_hits["instance_id"] == 0xFFFFFFFF, ref[:count]["instance_id"] == 0xFFFFFFFF)


@pytest.mark.parametrize("blocks", [7, 8])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_frames_at_launch_shapes(gpu_ctx, blocks, off):
    """Frames of two paths per resident warp, at the seven blocks per SM of the opaque
    binary form and the eight of the others: both layouts give the same sums."""
    import torch
    from rustracer_gb300 import gbrt
    sd = scenes.icosphere_scene(subdiv=3)
    sc = gbrt.Scene(gpu_ctx, sd)
    width = 8 * blocks * torch.cuda.get_device_properties(0).multi_processor_count + off
    ubo = sd.ubo(width, 1, samples=1, bounces=4, exposure=1.0)
    out = []
    for layout in (8, 2):
        sc.set_tuning(layout)
        acc = gbrt.Accum(gpu_ctx, width, 1)
        sc.render(ubo, acc, mode=gbrt.MODE_WAVEFRONT)
        out.append(acc.download())
    assert out[0][..., :3].max() > 0
    assert np.array_equal(out[0], out[1])
