"""GPU build at the edges of its tiles (radix-sort tiles of 4,096, clustering
tiles, eight lanes per wide node): hits exact against the oracle, and the tree
does not depend on the order the triangles come in (distinct centroid codes
sort to one order, so a misplaced pair would show as another tree)."""
import numpy as np
import pytest

import oracle as O
from foundation_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(built):
    import foundation_gb300 as fg
    c = fg.Context(0)
    yield c
    c.close()


BUILDS = [dict(), dict(sah_collapse=True), dict(cluster=True), dict(cluster=True, sah_collapse=True),
          dict(cluster=True, cluster_radius=64), dict(sah_collapse=True, node_width=3)]


@pytest.mark.parametrize("n", [1, 2, 3, 9, 33, 255, 257, 2049, 4095, 4096, 4097, 8193, 70001])
def test_tree_and_hits(ctx, n):
    sc = S.soup_scene(n, seed=11)
    perm = np.random.default_rng(n).permutation(n)
    rays = S.incoherent_rays(3000, (0, 0, 0), (1, 1, 1), seed=4)
    want = O.OracleBVH(sc.verts, sc.idx).closest(rays)
    for opts in BUILDS:
        a = ctx.upload(sc.verts, sc.idx, gpu_build=True, **opts)
        b = ctx.upload(sc.verts, sc.idx[perm], gpu_build=True, **opts)
        ia, ib = a.info(), b.info()
        for k in ("num_wide_nodes", "num_leaves", "wide_depth", "num_refs", "sah_cost"):
            assert ia[k] == ib[k], (opts, k)
        h = a.closest(rays)
        assert np.array_equal(h["prim"], want["prim"]) and np.array_equal(h["t"].view(np.uint32), want["t"].view(np.uint32))
        hb = b.closest(rays)
        hit = hb["prim"] != 0xFFFFFFFF
        assert np.array_equal(hb["t"].view(np.uint32), want["t"].view(np.uint32))
        assert np.array_equal(perm[hb["prim"][hit]], want["prim"][hit])
        a.close()
        b.close()


def test_equal_codes(ctx):
    """Triangles with one centroid: the order among equal codes is the input
    order (Karras breaks ties by position), the hits are exact."""
    rng = np.random.default_rng(2)
    n = 5000
    e = rng.normal(size=(n, 3, 3)).astype(np.float32) * 0.05
    v = (e - 0.5 * (e.min(1, keepdims=True) + e.max(1, keepdims=True)) + 0.5).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    rays = S.incoherent_rays(2000, (0.3, 0.3, 0.3), (0.7, 0.7, 0.7), seed=4)
    s = ctx.upload(v.reshape(-1, 3), idx, gpu_build=True, sah_collapse=True)
    h, want = s.closest(rays), O.OracleBVH(v.reshape(-1, 3), idx).closest(rays)
    assert np.array_equal(h["prim"], want["prim"]) and np.array_equal(h["t"].view(np.uint32), want["t"].view(np.uint32))
    s.close()


def test_pool_reuse_and_return(built):
    """Builds share a context's pool: a live scene keeps its arrays while others
    come and go (also while the cache trains on one), and closing the context
    gives the memory back."""
    import torch
    import foundation_gb300 as fg
    torch.cuda.synchronize()
    a, b = S.soup_scene(40000, seed=1), S.soup_scene(150000, seed=2)
    rays = S.incoherent_rays(2000, (0, 0, 0), (1, 1, 1), seed=4)
    want = O.OracleBVH(a.verts, a.idx).closest(rays)
    free = []
    for _ in range(2):  # the first pass also pays for what the process keeps (modules, local memory)
        with fg.Context(0) as c:
            keep = c.upload(a.verts, a.idx, gpu_build=True, cluster=True, sah_collapse=True)
            for k in range(3):
                other = c.upload(b.verts, b.idx, gpu_build=True, cluster=bool(k & 1), sah_collapse=True)
                if k == 1:
                    c.cache_create(other, train_paths=2000, train_steps=1, batch=512)
                    cam = dict(eye=(0.5, 0.5, 2.5), target=(0.5, 0.5, 0.5))
                    c.render(other, 64, 64, 1, cam, cache=True, train_only=True, sky=(1.0, 1.0, 1.0))
                other.close()
                h = keep.closest(rays)
                assert np.array_equal(h["prim"], want["prim"]) and np.array_equal(h["t"], want["t"])
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[1] < 16 << 20
