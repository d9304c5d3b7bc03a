"""A cache-training frame does not depend on what the gradient and optimiser
entry points ran before it. A step adds a tenth of its gradient to the first
moment; two clean caches of one seed differ in it by the order of their samples
only (some per cent), while the gradient call before the third one's second
frame is many times as large (targets of 1e6). Bound: a difference of less than
the moment's own norm."""
import numpy as np
import pytest

import oracle as O
from foundation_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _moment(tmp_path, before):
    import foundation_gb300 as fg
    cs = S.cornell_scene(num_spheres=20, level=2)
    with fg.Context(0) as ctx:
        s = ctx.upload(cs.verts, cs.idx)
        s.set_materials(cs.tri_material, S.material_records(cs))
        s.set_lights(S.light_records(cs))
        ctx.cache_create(s, train_paths=16384, train_steps=1, batch=8192, seed=5)
        ctx.render(s, 48, 27, 1, S.CORNELL_CAMERA, seed=1, cache=True, train_only=True)
        before(ctx)
        ctx.render(s, 48, 27, 1, S.CORNELL_CAMERA, seed=2, cache=True, train_only=True)
        p = tmp_path / "cache.bin"
        ctx.cache_save(p)
        w, m, v = np.frombuffer(p.read_bytes()[44:], np.float32).reshape(3, -1)
        assert len(m) == O.mlp_num_params() and ctx.cache_stats()["steps"] == 2
        s.close()
        return m.copy()


def _large_gradient(ctx, offset):
    """A gradient call whose result buffer lies `offset` past a 16-byte boundary
    (0: written in place where the device can, 4: copied)."""
    import ctypes as C
    from foundation_gb300 import rt
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (300, 96)).astype(np.float32)
    t = np.full((300, 3), 1e6, np.float32)
    room = np.zeros(O.mlp_num_params() + 8, np.float32)
    at = (-room.ctypes.data % 16 + offset) // 4
    g = room[at:at + O.mlp_num_params()]
    loss = C.c_double()
    assert rt.load().fnd_rt_cache_gradient(ctx._h, x.ctypes.data, t.ctypes.data, 300, g.ctypes.data, C.byref(loss)) == 0
    assert np.linalg.norm(g) > 1e3


def test_gradient_call_leaves_nothing_behind(built, tmp_path):
    clean, again = _moment(tmp_path, lambda c: None), _moment(tmp_path, lambda c: None)
    assert np.linalg.norm(again - clean) < np.linalg.norm(clean)
    for offset in (0, 4):
        after = _moment(tmp_path, lambda c: _large_gradient(c, offset))
        assert np.linalg.norm(after - clean) < np.linalg.norm(clean), offset
