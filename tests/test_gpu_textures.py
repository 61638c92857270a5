"""Texture filtering on the any-hit path against the oracle, bit for bit."""
import numpy as np
import pytest

from rustracer_gb300 import scenes, types as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (5, 7), (8, 4), (3, 16)])
@pytest.mark.parametrize("fmt", [T.TEX_RGBA8_UNORM, T.TEX_RGBA8_SRGB, T.TEX_RGBA16F])
def test_alpha_texture_wrap_modes(gpu_ctx, size, fmt):
    """Alpha-tested hits through textures of every wrap mode, at sizes that are
    powers of two and not, with uv on both sides of zero: the opacity decides
    the hit, so a texel off shows."""
    from rustracer_gb300 import gbrt
    import pyoracle as O
    rng = np.random.default_rng(size[0] * 31 + size[1] + fmt)
    w, h = size
    wraps = [T.WRAP_REPEAT, T.WRAP_CLAMP_TO_EDGE, T.WRAP_MIRRORED_REPEAT]
    b, tex = scenes.GeoBuilder(), []
    for k in range(9):  # a layer of triangles per pair of wrap modes, one behind the other
        if fmt == T.TEX_RGBA16F:
            img = rng.random((h, w, 4)).astype(np.float16).view(np.uint16)
        else:
            img = rng.integers(0, 256, (h, w, 4)).astype(np.uint8)
        tex.append((w, h, fmt, wraps[k % 3], wraps[k // 3], img))
        m = scenes.lambert((0.5, 0.5, 0.5))
        m["alpha_mode"] = T.ALPHA_MASK
        m["alpha_cutoff"] = 0.5
        m["base_color_texture"] = (k, 0)
        n = 40
        c = rng.uniform(-1, 1, (n, 1, 3)) * (1, 1, 0) + (0, 0, -0.1 * k)
        p = (c + rng.normal(0, 0.3, (n, 3, 3)) * (1, 1, 0)).reshape(-1, 3)
        b.add_mesh(p.astype(np.float32), np.arange(3 * n).reshape(-1, 3), b.add_material(m),
                   np.tile([0, 0, 1.0], (3 * n, 1)).astype(np.float32),
                   uv=rng.uniform(-3, 3, (3 * n, 2)).astype(np.float32))
    sd = b.finish(textures=tex, camera=dict(eye=(0, 0, 3), direction=(0, 0, -1), fov_deg=60.0), name="wraps")
    rays = np.zeros(4000, T.RAY)
    rays["org"] = np.column_stack([rng.uniform(-1, 1, (4000, 2)), np.full(4000, 2.0)])
    rays["dir"] = (0.0, 0.0, -1.0)
    rays["tmax"] = 1e4
    ref, _ = O.OracleScene(sd).trace(rays)
    hits, _ = gbrt.Scene(gpu_ctx, sd).trace(rays)
    assert len(np.unique(ref["custom_index"])) > 2  # several layers show
    for f in ("instance_id", "primitive_id", "t", "u", "v"):
        assert np.array_equal(hits[f], ref[f]), f
