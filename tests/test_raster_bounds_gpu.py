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


# vertices 300,000 pixels and more off the target
FAR = [(-251.3, -203.7), (249.1, -197.9), (3.7, 311.3)]


def _cancelling(far, persp):
    """Coordinates of magnitude `far` whose interpolated value is about 0 in the
    middle of the target."""
    p = np.array(FAR, np.float32).astype(np.float64)
    w = 1 + np.float32(persp) * p[:, 0]
    b = np.linalg.solve(np.vstack([(p / w[:, None]).T, np.ones(3)]), [0, 0, 1.0]) / w
    uv = np.random.default_rng(3).uniform(-1, 1, (3, 2)) * far
    uv[2] = -(b[0] * uv[0] + b[1] * uv[1]) / b[2]
    return uv


@pytest.mark.parametrize("shape,far", [((512, 512), 1e6), ((64, 4096), 1e6), ((16384, 16), 3e4), ((512, 512), 1e8),
                                       ((37, 53), 1e9)])
def test_far_coordinates(built, shape, far):
    _draw(2048, 2048, shape, FAR, _cancelling(far, 0.0019), 0.0019)
