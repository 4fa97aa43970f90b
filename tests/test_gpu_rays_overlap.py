"""Host ray batches whose result arrays lie over the rays, or over one
another: the rays are read as they were at the call, and the results are
stored in the order t, u, v, prim_id."""
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


def aligned(bytes_, offset):
    """Bytes that start `offset` past a 16-byte boundary."""
    buf = np.empty(bytes_ + 64, np.uint8)
    first = -buf.ctypes.data % 16 + offset
    return buf[first:first + bytes_]


def ptr(a, byte=0):
    return C.c_void_p(a.ctypes.data + byte)


@pytest.mark.parametrize("offset", [0, 4])
@pytest.mark.parametrize("n", [1, 33, 3000, 300001])
def test_results_over_the_rays(scene, n, offset):
    rays = make_rays(n, n)
    want = scene.trace_closest(rays, wavefront=True)
    occ_want = scene.trace_any(rays, wavefront=True)
    lib, ctx = scene.ctx.lib, scene.ctx
    buf = aligned(32 * n, offset)
    for first in (0, 16 * n):   # the results over the first or the second half of the rays
        buf[:] = rays.view(np.uint8).ravel()
        ctx.check(lib.dl_trace_closest(scene.h, ptr(buf), n, *(ptr(buf, first + 4 * n * k) for k in range(4))))
        got = buf[first:first + 16 * n].reshape(4, -1)
        assert np.array_equal(got[0].view(np.int32), want[0])
        for k in (1, 2, 3):
            assert np.array_equal(got[k].view(np.float32), want[k])
    for first in (0, 3):        # 3: over the high bytes of the rays' origins
        buf[:] = rays.view(np.uint8).ravel()
        ctx.check(lib.dl_trace_any(scene.h, ptr(buf), n, ptr(buf, first)))
        assert np.array_equal(buf[first:first + n], occ_want)


@pytest.mark.parametrize("offset", [0, 1])   # written by the kernel, copied
def test_results_over_one_another(scene, offset):
    n = 5000
    rays = make_rays(n, 7)
    want = scene.trace_closest(rays, wavefront=True)
    lib, ctx = scene.ctx.lib, scene.ctx
    one, two = aligned(4 * n, offset), aligned(4 * n, offset)
    ctx.check(lib.dl_trace_closest(scene.h, ptr(rays), n, ptr(one), ptr(one), ptr(one), ptr(one)))
    assert np.array_equal(one.copy().view(np.int32), want[0])
    ctx.check(lib.dl_trace_closest(scene.h, ptr(rays), n, ptr(one), ptr(two), ptr(two), ptr(two)))
    assert np.array_equal(two.copy().view(np.float32), want[3])
    assert np.array_equal(one.copy().view(np.int32), want[0])
