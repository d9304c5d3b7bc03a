"""The raster pass where its quick evaluation turns to the defining one: bytes
equal to the scalar restatement for colours beyond [0, 1], colours and texels
that land on rounding boundaries, textures of one texel and of more than
16,384 texels a side, coordinates far outside the repeat, large and tiny
triangles, widths that are no multiple of the pixels per thread, and target
rows off the 16-byte boundary."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _draw(W, H, verts, tex, persp=0.0, clear=(0.1, 0.5, 1.5, -0.2), device=False):
    import torch
    import foundation_gb300 as fg
    from foundation_gb300 import rt
    eye = np.eye(4, dtype=np.float32).ravel(order="F")
    proj = eye.copy()
    proj[3] = persp
    idx = np.arange(len(verts), dtype=np.uint16)
    want = O.raster_draw(W, H, eye, eye, proj, tex, verts.view(np.float32).reshape(-1, 7), idx, clear=clear,
                         cull_back=False)
    with fg.Context(0) as ctx:
        got = ctx.raster_draw(W, H, eye, eye, proj, tex, verts, idx, clear=clear, cull_back=False)
        if device:
            dev = torch.zeros(4 * W * H + 4, dtype=torch.uint8, device="cuda")[4:]
            ctx.raster_draw(W, H, eye, eye, proj, tex, verts, idx, clear=clear, cull_back=False, out=dev)
            ctx.sync()
            assert np.array_equal(dev.cpu().numpy().reshape(H, W, 4), want)
    assert np.array_equal(got, want), int((got != want).any(-1).sum())


def _verts(n, seed, scale, color, uv):
    from foundation_gb300 import rt
    rng = np.random.default_rng(seed)
    v = np.zeros(3 * n, rt.RASTER_VERTEX_DTYPE)
    v["pos"] = rng.uniform(-1.2, 1.2, (n, 1, 2)).repeat(3, 1).reshape(-1, 2) + rng.uniform(-scale, scale, (3 * n, 2))
    v["color"] = rng.uniform(*color, (3 * n, 3))
    v["uv"] = rng.uniform(*uv, (3 * n, 2))
    return v


@pytest.mark.parametrize("W,H", [(1, 1), (3, 5), (64, 33), (257, 130), (512, 64)])
@pytest.mark.parametrize("case", ["plain", "bright", "far_uv", "tiny", "huge"])
def test_bytes(built, W, H, case):
    rng = np.random.default_rng(W)
    tex = rng.integers(0, 256, (37, 53, 4), dtype=np.uint8)
    v = {"plain": _verts(25, 1, 0.7, (0, 1), (0, 1)), "bright": _verts(25, 2, 0.7, (-4, 4), (-2, 3)),
         "far_uv": _verts(25, 3, 0.7, (0, 1), (-3000, 3000)), "tiny": _verts(400, 4, 0.01, (0, 1), (0, 1)),
         "huge": _verts(6, 5, 900.0, (0, 1), (0, 2))}[case]
    _draw(W, H, v, tex, persp=0.0 if case == "huge" else 0.3, device=True)


@pytest.mark.parametrize("shape", [(1, 1), (2, 16385), (3, 2)])
def test_textures_and_ties(built, shape):
    """Flat colours of k / 510 under a white texel sit on rounding boundaries."""
    from foundation_gb300 import rt
    h, w = shape
    tex = np.full((h, w, 4), 255, np.uint8)
    if h == 3:
        tex[:] = np.random.default_rng(1).integers(0, 256, tex.shape)
    v = np.zeros(3 * 40, rt.RASTER_VERTEX_DTYPE)
    for k in range(40):
        x = -1 + 0.05 * k
        v["pos"][3 * k:3 * k + 3] = [(x, -1), (x + 0.05, -1), (x, 1)]
        v["color"][3 * k:3 * k + 3] = ((2 * k + 1) / 510.0, k / 255.0, (254 - k) / 510.0)
        v["uv"][3 * k:3 * k + 3] = [(0, 0), (1, 0), (0, 1)]
    _draw(200, 90, v, tex)


def test_not_finite(built):
    """Infinite and NaN vertex colours and coordinates take the definition."""
    v = _verts(9, 8, 0.8, (0, 1), (0, 1))
    v["color"][1] = np.inf
    v["color"][4, 1] = np.nan
    v["uv"][7] = np.nan
    v["uv"][10] = np.inf
    _draw(65, 40, v, np.random.default_rng(1).integers(0, 256, (8, 8, 4), dtype=np.uint8))


@pytest.mark.parametrize("nv,ni", [(3, 0), (3, 3), (64, 126), (64, 129), (65, 126), (66, 66), (300, 600)])
def test_mesh_sizes(built, nv, ni):
    """Meshes that travel with the launch (up to 64 vertices and 128 indices)
    and ones that are copied, with shared and unused vertices; bright colours
    take the paths that read the vertices again."""
    import foundation_gb300 as fg
    rng = np.random.default_rng(nv + ni)
    tex = rng.integers(0, 256, (7, 5, 4), dtype=np.uint8)
    v = _verts((nv + 2) // 3, 6, 0.8, (-3, 3), (-2, 3))[:nv]
    idx = rng.integers(0, nv, ni).astype(np.uint16)
    eye = np.eye(4, dtype=np.float32).ravel(order="F")
    want = O.raster_draw(97, 41, eye, eye, eye, tex, v.view(np.float32).reshape(-1, 7), idx, clear=(0.2, 0.4, 0.6, 1.0),
                         cull_back=False)
    with fg.Context(0) as ctx:
        for _ in range(2):
            got = ctx.raster_draw(97, 41, eye, eye, eye, tex, v, idx, clear=(0.2, 0.4, 0.6, 1.0), cull_back=False)
            assert np.array_equal(got, want)
