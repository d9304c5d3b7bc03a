"""The traversal's own checks in the kernels that an application reaches: every
query on an uploaded scene (triangle records) whose device copy has been given a
child index or a triangle range past its arrays, or an instance id past the
instances, ends with the bad-index code and no access out of range, through the
helping loop alone (few rays), both loops (many), statistics, batches, two
levels, and the path kernels of renders and cache training; the restored scene
then answers as before. (test_status_word.py drives the plain forms and the
kernels over vertex planes.) Chains past and within the stack run through the
record kernels by hand-made scenes: no upload accepts the former."""
import ctypes as C
import os

import numpy as np
import pytest

from foundation_gb300 import scenes as S
from test_status_word import CASES, FND_ERR_INVALID_SCENE, NODE, STACK_OVERFLOW, TRI_ID, _rays

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
FEW, MANY = 500, 200000  # (the second loop alone takes up to 116,736)
PAST = 1 << 30


@pytest.fixture(scope="module")
def L(built):
    lib = C.CDLL(os.path.join(HERE, "_build", "libproduct_check.so"))
    P = C.c_void_p
    lib.product_scene_bytes.argtypes = [P, C.c_int, C.c_int, P]
    lib.product_trace_records.argtypes = [P, C.c_uint32, P, C.c_uint32, P, C.c_uint32, C.c_int, P, P]
    return lib


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _get(L, scene, part):
    a = np.zeros(scene.info()["node_bytes" if part == 0 else "tri_bytes"], np.uint8)
    assert L.product_scene_bytes(scene.handle, part, 0, _p(a)) == 0
    return a


def _corrupt(nodes, case):
    n = nodes.copy().view(NODE)
    if case == "child":
        n["child_base"][0] = PAST
    else:
        leaf = np.nonzero((n["meta"] & 0x80).any(1))[0]
        assert len(leaf)
        n["tri_base"][leaf[::2]] = PAST  # (every second: most paths go on to the tail)
    return n.view(np.uint8)


def _queries(ctx, scene, two):
    """name -> call; each call's error is the device status's."""
    import torch
    import foundation_gb300 as fg
    from foundation_gb300 import rt
    rays = {n: S.incoherent_rays(n, (-1, 0, -1), (1, 2, 1), seed=3) for n in (FEW, MANY)}
    dev = {n: torch.from_numpy(r).cuda() for n, r in rays.items()}
    cam = S.CORNELL_CAMERA

    def batch(n):
        a, b = torch.zeros(2 * n, dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda")
        job = fg.Batch(ctx, [(scene, dev[n], a, rt.QUERY_CLOSEST), (scene, dev[n], b, rt.QUERY_ANY)])
        try:
            job.launch()
            ctx.sync()
        finally:
            job.close()
        return a.cpu().numpy(), b.cpu().numpy()

    q = {}
    for n in (FEW, MANY):
        q[f"closest {n}"] = lambda n=n: (scene.closest(rays[n]),)
        q[f"any {n}"] = lambda n=n: (scene.any(rays[n]),)
        if not two:
            q[f"statistics {n}"] = lambda n=n: scene.closest(rays[n], stats=True)[:1]
            q[f"batch {n}"] = lambda n=n: batch(n)
    for name, kw in (("tail", {}), ("wavefront", dict(wavefront=True))):
        q["render " + name] = lambda kw=kw: ctx.render(scene, 64, 36, 1, cam, sky=(1, 1, 1), seed=2, **kw)

    def train():
        ctx.render(scene, 64, 36, 1, cam, sky=(1, 1, 1), seed=2, cache=True, train_only=True)
        ctx.sync()

    q["training"] = train
    return q


def _run(L, ctx, scene, two, edits):
    import foundation_gb300 as fg
    queries = _queries(ctx, scene, two)
    before = {k: f() for k, f in queries.items()}
    for holder, part, good, bad in edits:
        assert L.product_scene_bytes(holder.handle, part, 1, _p(np.ascontiguousarray(bad))) == 0
        for k, f in queries.items():
            with pytest.raises(fg.FndError) as e:
                f()
            assert e.value.code == FND_ERR_INVALID_SCENE, k
        assert L.product_scene_bytes(holder.handle, part, 1, _p(good)) == 0
        for k, f in queries.items():
            after = f()
            if not k.startswith(("render", "training")):
                for a, b in zip(before[k], after):
                    assert np.array_equal(a, b), k


def test_one_level(L):
    import foundation_gb300 as fg
    sc = S.cornell_scene(num_spheres=8, level=2)
    with fg.Context(0) as ctx:
        scene = ctx.upload(sc.verts, sc.idx)
        ctx.cache_create(scene, train_paths=8192, train_steps=1, batch=1024, seed=1)
        nodes = _get(L, scene, 0)
        _run(L, ctx, scene, False, [(scene, 0, nodes, _corrupt(nodes, c)) for c in ("child", "range")])
        scene.close()


def test_two_levels(L):
    import foundation_gb300 as fg
    sc = S.cornell_scene(num_spheres=8, level=2)
    with fg.Context(0) as ctx:
        blas = ctx.upload(sc.verts, sc.idx, margin_scale=64)
        move = np.eye(3, 4, dtype=np.float32)
        inst = []
        for k in range(64):  # (a top level of several nodes)
            m = move.copy()
            m[0, 3] = 0.01 * k
            inst.append((blas, m, 100000 * k))
        scene = ctx.instances(inst)
        ctx.cache_create(scene, train_paths=8192, train_steps=1, batch=1024, seed=1)
        bottom, top, ids = _get(L, blas, 0), _get(L, scene, 0), _get(L, scene, 1)
        bad_ids = ids.copy().view(np.uint32).reshape(-1, 12)
        bad_ids[:, 3] = PAST
        edits = [(blas, 0, bottom, _corrupt(bottom, c)) for c in ("child", "range")]
        edits += [(scene, 0, top, _corrupt(top, c)) for c in ("child", "range")]
        edits.append((scene, 1, ids, bad_ids.view(np.uint8)))
        _run(L, ctx, scene, True, edits)
        scene.close()
        blas.close()


@pytest.mark.parametrize("any_hit", [0, 1], ids=["closest", "any"])
def test_chains(L, any_hit):
    """Deeper than the stack: each of many rays overflows in the first loop (with
    few, lanes that help keep the stacks short). Within it: the hit, both ways."""
    for case, ns, want in (("stack_overflow", (MANY,), STACK_OVERFLOW), ("deep_but_fits", (FEW, MANY), 0)):
        mk_nodes, mk_planes, _, hit = CASES[case]
        nodes, planes = mk_nodes(), mk_planes()
        tris = np.ascontiguousarray(planes.transpose(1, 0, 2))
        for n in ns:
            rays = _rays(n)
            out = np.zeros(n, np.uint8) if any_hit else np.zeros((n, 2), np.uint32)
            st = np.zeros(1, np.uint32)
            assert L.product_trace_records(_p(nodes), len(nodes), _p(tris), len(tris), _p(rays), n, any_hit, _p(out),
                                           _p(st)) == 0
            assert int(st[0]) == want, (case, n)
            if any_hit:
                assert (out == (1 if hit else 0)).all()
            else:
                assert (out[:, 0] == (TRI_ID if hit else 0xFFFFFFFF)).all()
