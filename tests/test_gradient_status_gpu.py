"""A gradient call reports the status word: a tensor-core wait that gave up (the
word is set from the host in its place) ends the call with the timeout code, not
with FND_OK and a partial gradient. The word is clear for the next call."""
import ctypes as C
import os

import numpy as np
import pytest

from foundation_gb300 import scenes as S

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
STATUS_TIMEOUT = 2
FND_ERR_TIMEOUT = -7


@pytest.mark.parametrize("offset", [0, 4], ids=["in place", "copied"])
def test_gradient_reports_a_timeout(built, offset):
    import foundation_gb300 as fg
    from foundation_gb300 import rt
    L = C.CDLL(os.path.join(HERE, "_build", "libproduct_check.so"))
    L.product_latch_status.argtypes = [C.c_void_p, C.c_uint32]
    sc = S.cornell_scene(num_spheres=2, level=1)
    with fg.Context(0) as ctx:
        scene = ctx.upload(sc.verts, sc.idx)
        ctx.cache_create(scene, seed=3)
        room = np.zeros(200 * 96 + 8, np.float32)
        at = (-room.ctypes.data % 16 + offset) // 4
        x = room[at:at + 200 * 96]
        x[:] = np.random.default_rng(1).uniform(-1, 1, x.size)
        t = np.full((200, 3), 0.5, np.float32)
        g, loss = np.zeros(22720, np.float32), C.c_double()
        call = lambda: rt.load().fnd_rt_cache_gradient(ctx._h, x.ctypes.data, t.ctypes.data, 200,  # noqa: E731
                                                       g.ctypes.data, C.byref(loss))
        assert call() == 0
        assert L.product_latch_status(ctx._h, STATUS_TIMEOUT) == 0
        assert call() == FND_ERR_TIMEOUT
        assert call() == 0 and loss.value > 0
        scene.close()
