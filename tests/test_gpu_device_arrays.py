"""Entry points that read the caller's arrays in place, given device memory
where they expect host memory: the host must not touch it.  The calls copy it
and give the results they give for host arrays."""
import ctypes as C

import numpy as np
import pytest
import torch

from drawlab_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def ptr(a):
    return C.c_void_p(a.data_ptr() if isinstance(a, torch.Tensor) else a.ctypes.data)


@pytest.fixture(scope="module")
def ctx():
    return api.Context(0)


def on_device(shape, dtype):
    t = torch.empty(shape, dtype=dtype, device="cuda:0")
    torch.cuda.synchronize()
    return t


def test_ray_batches(ctx):
    s = api.Scene.from_data(ctx, scenes.cornell(16, 16))
    r = np.random.default_rng(1)
    n = 1001
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = r.uniform(-0.9, 0.9, (n, 3))
    rays[:, 3] = 1e-4
    rays[:, 4:7] = r.normal(size=(n, 3))
    rays[:, 7] = r.uniform(0.1, 2.0, n)
    want = s.trace_closest(rays)
    occ_want = s.trace_any(rays)
    d_rays = torch.from_numpy(rays).to("cuda:0")
    d_out = [on_device(n, torch.int32)] + [on_device(n, torch.float32) for _ in range(3)]
    h_out = [np.empty(n, np.int32)] + [np.empty(n, np.float32) for _ in range(3)]
    for rin in (rays, d_rays):
        for outs in (h_out, d_out):
            ctx.check(ctx.lib.dl_trace_closest(s.h, ptr(rin), n, *(ptr(o) for o in outs)))
            for o, w in zip(outs, want):
                assert np.array_equal(o.cpu().numpy() if isinstance(o, torch.Tensor) else o, w)
        occ, d_occ = np.full(n, 9, np.uint8), on_device(n, torch.uint8)
        ctx.check(ctx.lib.dl_trace_any(s.h, ptr(rin), n, ptr(occ)))
        ctx.check(ctx.lib.dl_trace_any(s.h, ptr(rin), n, ptr(d_occ)))
        assert np.array_equal(occ, occ_want) and np.array_equal(d_occ.cpu().numpy(), occ_want)


def test_network_inputs(ctx):
    g = api.Guide(ctx, seed=4)
    x = np.random.default_rng(2).random((300, 6)).astype(np.float32)
    want = g.forward(x)
    d_x, d_y, y = torch.from_numpy(x).to("cuda:0"), on_device((300, 40), torch.float32), np.empty((300, 40), np.float32)
    ctx.check(ctx.lib.dl_guide_forward(g.h, 300, ptr(d_x), ptr(y)))
    ctx.check(ctx.lib.dl_guide_forward(g.h, 300, ptr(d_x), ptr(d_y)))
    assert np.array_equal(y, want) and np.array_equal(d_y.cpu().numpy(), want)
