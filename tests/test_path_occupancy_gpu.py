"""The path kernels (tail, training paths) of one-level scenes keep 16 warps per
SM: what bounds them is the latency of their longest paths, and a branch that
only ray batches need, compiled into them, once took them from 128 registers a
thread to 168 and so to 12 warps."""
import ctypes as C
import os

import numpy as np
import pytest

from foundation_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def test_path_kernels_keep_their_warps(built):
    import foundation_gb300 as fg
    L = C.CDLL(os.path.join(os.path.dirname(os.path.abspath(__file__)), "_build", "libproduct_check.so"))
    with fg.Context(0):
        assert L.product_tail_blocks(0) >= 4
        assert L.product_training_blocks(0) >= 4
        assert L.product_tail_blocks(1) >= 3 and L.product_training_blocks(1) >= 3


@pytest.mark.parametrize("width,height", [(384, 304), (400, 300), (480, 270), (456, 341), (457, 341)])
def test_automatic_threshold(built, width, height):
    """Waves around the sizes where the automatic threshold changes (768 and
    1,024 paths per SM: 116,736 and 155,648 on the full chip): the rays of the
    wavefront stages, and their image up to the order of at most 8 x 3
    non-negative FP32 additions (2^-24 each)."""
    import foundation_gb300 as fg
    cs = S.cornell_scene(num_spheres=20, level=2)
    with fg.Context(0) as ctx:
        s = ctx.upload(cs.verts, cs.idx)
        s.set_materials(cs.tri_material, S.material_records(cs))
        s.set_lights(S.light_records(cs))
        img, counts = [], []
        for kw in ({}, dict(wavefront=True)):
            img.append(ctx.render(s, width, height, 1, S.CORNELL_CAMERA, seed=4, **kw))
            st = ctx.render_stats()
            counts.append((st["extension_rays"], st["shadow_rays"]))
        assert counts[0] == counts[1]
        np.testing.assert_allclose(img[0], img[1], rtol=24 * 2.0 ** -24, atol=0)
        s.close()
