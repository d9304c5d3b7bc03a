"""The traversal kernels' per-warp ring of waiting triangles, at the sizes
where it turns: no triangles at all, leaves of one triangle, nodes whose
leaves fill the ring many times over in one step (coincident triangles, which
no box separates), ray counts around one warp, and every threshold of the
launch shape that decides when a part-filled ring is tested. Exact against
the oracle: the order of the tests must not show."""
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


def _geometry(kind):
    rng = np.random.default_rng(3)
    if kind == "one":
        v = np.array([[0.0, 0, 0.5], [1, 0, 0.5], [0, 1, 0.5]], np.float32)
    elif kind == "stack":  # 300 coincident copies, then 300 shifted along z
        t = np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]])
        v = np.concatenate([t + [0, 0, 0.25 if k < 300 else k * 1e-3] for k in range(600)]).astype(np.float32)
    else:
        return S.soup_scene(3000, seed=5)
    return S.Scene(v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3))


def _rays(n):
    rays = S.incoherent_rays(n, (0, 0, 0), (1, 1, 1), seed=9)
    rays[::5, 4:7] = (0.01, 0.02, 1.0)  # through the stacked triangles
    rays[::7, 7] = 0.3
    return rays


@pytest.mark.parametrize("kind", ["one", "stack", "soup"])
@pytest.mark.parametrize("n", [1, 31, 33, 5000])
def test_ring_matches_oracle(ctx, kind, n):
    sc, rays = _geometry(kind), _rays(n)
    b = O.OracleBVH(sc.verts, sc.idx)
    want, want_any = b.closest(rays), b.any(rays)
    builds = [{}, {"spatial_splits": True, "sah_collapse": True}]
    if kind != "stack":  # clustering coincident triangles gives a chain deeper than the stack, which upload refuses
        builds.append({"gpu_build": True, "cluster": True})
    for opts in builds:
        scene = ctx.upload(sc.verts, sc.idx, **opts)
        for refill in (1, 8, 32):
            for wait in (0, 1, 32):
                ctx.set_trace_config(short_stack=4, refill_min=refill, postpone_min=wait)
                h = scene.closest(rays)
                assert np.array_equal(h["prim"], want["prim"]), (opts, refill, wait)
                assert np.array_equal(h["t"].view(np.uint32), want["t"].view(np.uint32))
                assert np.array_equal(scene.any(rays), want_any)
        scene.close()
    ctx.set_trace_config()


@pytest.mark.parametrize("n", [2, 63, 300, 1217, 2433, 4865, 30000, 116735, 116736, 116737, 300001])
def test_small_batches(ctx, n):
    """Batches on few lanes per warp, around the sizes where the lane count and
    the grid change (1,216 blocks of four warps on the full chip), one- and
    two-level."""
    sc, rays = _geometry("soup"), _rays(n)
    b = O.OracleBVH(sc.verts, sc.idx)
    want, want_any = b.closest(rays), b.any(rays)
    scene = ctx.upload(sc.verts, sc.idx)
    two = ctx.instances([(scene, np.eye(3, 4, dtype=np.float32), 0)])
    for s in (scene, two):
        h = s.closest(rays)
        assert np.array_equal(h["prim"], want["prim"])
        assert np.array_equal(h["t"].view(np.uint32), want["t"].view(np.uint32))
        assert np.array_equal(s.any(rays), want_any)
    two.close()
    scene.close()


@pytest.mark.parametrize("n", [40, 3000, 116735, 116737, 200000])
def test_batches_of_scenes(ctx, n):
    """One launch over scenes of different size and both query kinds, on either
    side of the size from which a warp starts with all its lanes: lanes that
    help another lane's ray must take its scene and kind with it."""
    import torch
    import foundation_gb300 as fg
    jobs, want = [], []
    for k, kind in enumerate(("soup", "one", "stack", "soup")):
        sc, rays = _geometry(kind), _rays(max(1, n // 8))
        b = O.OracleBVH(sc.verts, sc.idx)
        scene = ctx.upload(sc.verts, sc.idx)
        rd = torch.from_numpy(rays).cuda()
        for q in (0, 1):
            out = torch.zeros(len(rays) * (1 if q else 2), dtype=torch.uint8 if q else torch.int32, device="cuda")
            jobs.append((scene, rd, out, q))
            want.append(b.any(rays) if q else b.closest(rays))
    torch.cuda.synchronize()
    batch = fg.Batch(ctx, jobs)
    batch.launch()
    ctx.sync()
    for (scene, rd, out, q), w in zip(jobs, want):
        got = out.cpu().numpy()
        if q:
            assert np.array_equal(got, w)
        else:
            got = got.view(np.uint32).reshape(-1, 2)
            assert np.array_equal(got[:, 0], w["prim"]) and np.array_equal(got[:, 1], w["t"].view(np.uint32))
    batch.close()
    for j in jobs[::2]:
        j[0].close()


@pytest.mark.parametrize("width,height", [(1, 1), (31, 1), (33, 1), (65, 3), (200, 7)])
@pytest.mark.parametrize("sun", [False, True])
def test_rays_of_a_warps_paths(ctx, width, height, sun):
    """The tail kernel traces the segments and shadow rays of a warp's paths
    together (part-filled warps, up to three rays per lane, lanes whose path
    has ended): the same rays as the wavefront stages, and the same image up to
    the order of at most 3 x 8 x 3 non-negative FP32 additions (2^-24 each)."""
    from foundation_gb300 import scenes as S
    cs = S.cornell_scene()
    s = ctx.upload(cs.verts, cs.idx)
    s.set_materials(cs.tri_material, S.material_records(cs))
    s.set_lights(S.light_records(cs))
    kw = dict(seed=9, sky=(0.1, 0.2, 0.3), rr_start=2)
    if sun:
        kw.update(sun_dir=(0.2, 0.4, 1.0), sun_irradiance=(0.5, 0.25, 0.75))
    got = []
    for opts in (dict(wavefront=True), dict(tail_paths=1 << 28)):
        img = ctx.render(s, width, height, 3, S.CORNELL_CAMERA, **kw, **opts)
        st = ctx.render_stats()
        got.append((img, st["extension_rays"], st["shadow_rays"]))
    assert got[0][1:] == got[1][1:]
    np.testing.assert_allclose(got[1][0], got[0][0], rtol=72 * 2.0 ** -24, atol=0)
    s.close()


@pytest.mark.parametrize("n", [1, 33, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, 3 << 19, (3 << 19) + 9])
@pytest.mark.parametrize("kind", ["pageable", "pinned", "rays off by 4 bytes", "hits off by 4 bytes", "overlap"])
def test_host_rays_in_place(ctx, n, kind):
    """Host rays are traced where they lie, and small batches' hits written
    there; past a size the hits are copied back, past another in two parts;
    unaligned buffers and ones that overlap take copies. All as from the
    device, to the bit."""
    import torch

    import foundation_gb300 as fg
    if kind == "overlap" and n > 1 << 19:
        pytest.skip("copied in parts: hits may land on rays that are still to be copied")
    sc = S.soup_scene(3000, seed=5)
    s = ctx.upload(sc.verts, sc.idx)
    rays = _rays(n)
    dev = torch.from_numpy(rays).cuda()
    want = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    occ = torch.empty(n, dtype=torch.uint8, device="cuda")
    s.closest(dev, want)
    s.any(dev, occ)
    ctx.sync()
    want, occ = want.cpu().numpy().view(np.uint32).reshape(n, 2), occ.cpu().numpy()
    dt = fg.rt.HIT_DTYPE
    if kind == "pinned":
        rb, hb = fg.rt.PinnedBuffer(32 * n), fg.rt.PinnedBuffer(8 * n)
        hr, out = rb.view(np.float32, (n, 8)), hb.view(dt, (n,))
    else:
        room = np.zeros(40 * n + 64, np.uint8)
        at = -room.ctypes.data % 16 + (4 if kind == "rays off by 4 bytes" else 0)
        hr = room[at:at + 32 * n].view(np.float32).reshape(n, 8)
        to = at + 32 * n + (-(at + 32 * n + room.ctypes.data)) % 8 + (4 if kind == "hits off by 4 bytes" else 0)
        out = (room[at:at + 8 * n] if kind == "overlap" else room[to:to + 8 * n]).view(dt)
    hr[:] = rays
    if kind != "overlap":
        got = np.full(n, 7, np.uint8)
        s.any(hr, got)
        assert (got == occ).all()
    s.closest(hr, out)
    assert (out["prim"] == want[:, 0]).all() and (out["t"].view(np.uint32) == want[:, 1]).all()
    s.close()
