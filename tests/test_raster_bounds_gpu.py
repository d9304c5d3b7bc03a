"""The error bounds of the raster pass's quick evaluations: textures whose
texels jump between 0 and 255, so that a texture coordinate's error shows at
its largest, on targets of millions of pixels, of which some lie within the
error of a rounding boundary. Bytes equal to the scalar restatement."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _draw(W, H, shape, corners, uv, persp):
    """One triangle over the whole target (corners in normalised device units
    before the perspective), a random 0 / 255 texture of shape (h, w)."""
    import foundation_gb300 as fg
    from foundation_gb300 import rt
    rng = np.random.default_rng(shape[0] + shape[1])
    tex = (rng.integers(0, 2, (*shape, 4)) * 255).astype(np.uint8)
    v = np.zeros(3, rt.RASTER_VERTEX_DTYPE)
    v["pos"] = corners
    v["color"] = rng.uniform(0.5, 1.0, (3, 3))
    v["uv"] = uv
    eye = np.eye(4, dtype=np.float32).ravel(order="F")
    proj = eye.copy()
    proj[3] = persp
    idx = np.arange(3, dtype=np.uint16)
    want = O.raster_draw(W, H, eye, eye, proj, tex, v.view(np.float32).reshape(-1, 7), idx, cull_back=False)
    with fg.Context(0) as ctx:
        got = ctx.raster_draw(W, H, eye, eye, proj, tex, v, idx, cull_back=False)
    assert np.array_equal(got, want), int((got != want).any(-1).sum())


SCREEN = [(-1.1, -1.2), (3.4, -1.1), (-1.0, 3.3)]


@pytest.mark.parametrize("shape", [(4096, 4096), (16, 16384), (16384, 16), (512, 512)])
def test_large_textures(built, shape):
    _draw(4096, 2048, shape, SCREEN, [(-0.93, -0.87), (0.97, -0.71), (-0.83, 1.07)], 0.1)
