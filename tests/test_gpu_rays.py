"""Host ray batches: sizes around a warp and a block, arrays the kernel reads
and writes in place and arrays it cannot (not 16-byte aligned), against the
renderer's own traversal kernels (bit-equal: the same tree, the same order)."""
import ctypes as C

import numpy as np
import pytest

from drawlab_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    ctx = api.Context(0)
    return api.Scene.from_data(ctx, scenes.material_spheres(64, 36, num_spheres=16, level=3))


def make_rays(n, seed):
    r = np.random.default_rng(seed)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = r.uniform((-20, 0.01, -20), (20, 3, 20), (n, 3))
    d = r.normal(size=(n, 3))
    rays[:, 3] = 1e-4
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = np.where(r.random(n) < 0.3, r.uniform(0.5, 10, n), np.inf)
    return rays


def at_offset(a, words):
    """A copy of `a` whose data starts `words` floats past a 16-byte boundary."""
    buf = np.empty(a.size + 8, a.dtype)
    start = (-(buf.ctypes.data // a.itemsize)) % (16 // a.itemsize) + words
    out = buf[start:start + a.size].reshape(a.shape)
    out[...] = a
    return out


@pytest.mark.parametrize("words", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 70001])
def test_host_ray_batches(scene, n, words):
    rays = make_rays(n, n)
    want = scene.trace_closest(rays, wavefront=True)
    occ_want = scene.trace_any(rays, wavefront=True)
    given = at_offset(rays, words)
    assert given.ctypes.data % 16 == 4 * words
    prim = at_offset(np.full(n, -7, np.int32), words)
    t, u, v = (at_offset(np.full(n, np.nan, np.float32), words) for _ in range(3))
    occ = np.full(n + 1, 9, np.uint8)[1:]
    p = [C.c_void_p(a.ctypes.data) for a in (given, prim, t, u, v, occ)]
    lib = scene.ctx.lib
    scene.ctx.check(lib.dl_trace_closest(scene.h, p[0], n, p[1], p[2], p[3], p[4]))
    scene.ctx.check(lib.dl_trace_any(scene.h, p[0], n, p[5]))
    for got, ref in zip((prim, t, u, v, occ), (*want, occ_want)):
        assert np.array_equal(got, ref)
    assert np.array_equal(given, rays)
