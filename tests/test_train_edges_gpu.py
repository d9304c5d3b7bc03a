"""The fused training kernel at the edges of its 128-row tiles, on features
that it reads in place (16-byte aligned) and on ones that are copied first,
against the FP64 oracle with BF16 rounding emulated (the bounds of
test_nrc_gpu.py; the same tile gives the same bits either way)."""
import numpy as np
import pytest

import oracle as O
from foundation_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(built):
    import foundation_gb300 as fg
    c = fg.Context(0)
    cs = S.cornell_scene(num_spheres=20, level=2)
    s = c.upload(cs.verts, cs.idx)
    c.cache_create(s, seed=3)
    yield c
    c.close()


def _at(a, offset):
    """A copy of a whose address is `offset` past a 16-byte boundary."""
    room = np.empty(a.nbytes + 32, np.uint8)
    at = -room.ctypes.data % 16 + offset
    out = room[at:at + a.nbytes].view(np.float32).reshape(a.shape)
    out[:] = a
    return out


@pytest.mark.parametrize("n", [1, 127, 128, 129, 300, 5000])
def test_gradient_edges(ctx, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 96)).astype(np.float32)
    t = rng.uniform(0, 2, (n, 3)).astype(np.float32)
    w = np.ascontiguousarray(ctx.cache_weights(), np.float32)
    u = w.view(np.uint32)
    bf = ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)
    _, loss_ref, g_ref = O.mlp_forward_backward(bf, x, t, emulate_bf16=True)
    got = [ctx.cache_gradient(_at(x, fx), _at(t, ft)) for fx, ft in ((0, 0), (4, 0), (0, 4))]
    for g, loss in got:
        assert abs(loss / loss_ref - 1) < 1e-2, (loss, loss_ref)
        off = 0
        for l in range(6):
            k = O.MLP_DIMS[l] * O.MLP_DIMS[l + 1]
            a, b = g[off:off + k], g_ref[off:off + k]
            assert np.linalg.norm(a - b) < 3e-2 * np.linalg.norm(b), l
            off += k
        if n <= 128:
            assert np.array_equal(g, got[0][0]) and loss == got[0][1]


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 255, 257, 3000])
def test_inference_edges(ctx, n):
    """A row's output depends on its own features only, whatever tile of 32 it
    lies in: the first rows of a large call, to the bit; and rows past the end
    are not written."""
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (4096, 96)).astype(np.float32)
    whole = ctx.cache_eval(x)
    assert np.array_equal(ctx.cache_eval(x[:n]), whole[:n])
    assert np.array_equal(ctx.cache_eval(x[7:7 + n]), whole[7:7 + n])
