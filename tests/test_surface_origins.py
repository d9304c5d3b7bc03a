"""Rays that start on a surface: t = 0 hits, whose sign is that of the rounding
of their plane, in a flat grid where up to six triangles of several nodes meet
at the origin. The lowest id wins and t keeps that triangle's own sign of zero,
also where the ray's length is a zero of either sign. CPU: the host compilation
of the node and triangle tests. GPU: batches (a few rays and many), one and two
levels. Exact against the brute-force oracle."""
import ctypes as C
import os

import numpy as np
import pytest

import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
CELLS = 32
DIRECTIONS = [(0.1, -1.0, 0.2), (0.1, 1.0, 0.2), (-0.3, -1.0, -0.2), (0.0, -1.0, 0.0)]


def _grid():
    k = np.arange(CELLS + 1)
    x, z = np.meshgrid(k / CELLS * 2 - 1, k / CELLS * 2 - 1, indexing="ij")
    v = np.stack([x.ravel(), np.zeros(x.size), z.ravel()], 1).astype(np.float32)
    i, j = np.meshgrid(np.arange(CELLS), np.arange(CELLS), indexing="ij")
    a = (i * (CELLS + 1) + j).ravel()
    b, c, d = a + 1, a + CELLS + 1, a + CELLS + 2
    f = np.stack([np.stack([a, c, b], 1), np.stack([b, c, d], 1)], 1).reshape(-1, 3)
    # ids out of spatial order, so that the lowest one is often tested last
    return v, np.ascontiguousarray(f[np.random.default_rng(7).permutation(len(f))], np.uint32)


def _rays(v, d, tmax):
    r = np.zeros((len(v), 8), np.float32)
    r[:, 0:3] = v
    r[:, 4:7] = d
    r[:, 7] = tmax
    return r


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _check(prim, tbits, want, what):
    assert (want["prim"] != 0xFFFFFFFF).mean() > 0.9, what
    assert np.array_equal(prim, want["prim"]), what
    assert np.array_equal(tbits, want["t"].view(np.uint32)), what


TMAX = [np.float32(np.inf), np.float32(0.0), np.float32(-0.0)]


@pytest.mark.parametrize("d", DIRECTIONS, ids=str)
def test_zero_distance_hits_emulated(built, d):
    L = C.CDLL(os.path.join(HERE, "_build", "libwide_emu.so"))
    P = C.c_void_p
    L.emu_build.restype = L.emu_instances.restype = P
    L.emu_build.argtypes = [P, C.c_uint32, P, C.c_uint32, C.c_uint32]
    L.emu_trace.argtypes = [P, P, C.c_uint64, P, C.c_int, P]
    L.emu_trace_single.argtypes = [P, P, C.c_uint64, P, C.c_int]
    L.emu_instances.argtypes = [P, P, P, C.c_uint32]
    L.emu_instances_trace.argtypes = [P, P, C.c_uint64, P, C.c_int]
    L.emu_free.argtypes = L.emu_instances_free.argtypes = [P]
    v, f = _grid()
    e = L.emu_build(_p(v), len(v), _p(f), len(f), 0)
    eye = np.eye(3, 4, dtype=np.float32)
    two = L.emu_instances(_p(np.array([e], np.uint64)), _p(eye), _p(np.zeros(1, np.uint32)), 1)
    for tmax in TMAX:
        rays = _rays(v, d, tmax)
        want = O.brute_closest(v, f, rays)
        out, st = np.zeros(2 * len(rays), np.uint32), np.zeros(4, np.uint64)
        L.emu_trace(e, _p(rays), len(rays), _p(out), 0, _p(st))
        _check(out[0::2], out[1::2], want, ("loop", tmax))
        L.emu_trace_single(e, _p(rays), len(rays), _p(out), 0)
        _check(out[0::2], out[1::2], want, ("single", tmax))
        L.emu_instances_trace(two, _p(rays), len(rays), _p(out), 0)
        _check(out[0::2], out[1::2], want, ("two levels", tmax))
    L.emu_instances_free(two)
    L.emu_free(e)


@pytest.mark.gpu
@pytest.mark.parametrize("d", DIRECTIONS, ids=str)
def test_zero_distance_hits_on_gpu(built, d):
    import foundation_gb300 as fg
    v, f = _grid()
    with fg.Context(0) as ctx:
        scenes = [ctx.upload(v, f, **o) for o in ({}, {"spatial_splits": True, "sah_collapse": True},
                                                  {"gpu_build": True, "cluster": True})]
        scenes.append(ctx.instances([(scenes[0], np.eye(3, 4, dtype=np.float32), 0)]))
        for tmax in TMAX:
            few = _rays(v, d, tmax)
            want = O.brute_closest(v, f, few)
            for n in (1, 128):  # 1,089 rays by the helping loop alone, 139,392 by both
                rays = np.tile(few, (n, 1))
                for k, s in enumerate(scenes):
                    h = s.closest(rays)
                    _check(h["prim"], h["t"].view(np.uint32),
                           {"prim": np.tile(want["prim"], n), "t": np.tile(want["t"], n)}, (k, n, tmax))
