"""Samples the film drops, and several contexts at once, on the resident kernel
and on a wavefront that it finishes, against the wavefront alone."""
import threading

import numpy as np
import pytest

from drawlab_gb300 import abi, api, scenes

pytestmark = pytest.mark.gpu

WAVEFRONT = dict(max_paths_in_flight=1 << 22)


@pytest.mark.parametrize("w,h,spp", [(64, 48, 3), (700, 500, 5)])   # one launch; finished
@pytest.mark.parametrize("bad", [-1.0, np.nan, np.inf])
def test_dropped_samples_are_counted(w, h, spp, bad):
    ctx = api.Context(0)
    data = scenes.cornell(w, h)
    for light in data.lights:
        light.radiance = (light.radiance[0], bad, light.radiance[2])
    s = api.Scene.from_data(ctx, data)
    a = s.render_film(abi.make_opts(spp=spp, max_depth=4, seed=2))
    na, ia = ctx.stats().invalid_samples, ctx.stats().iterations
    b = s.render_film(abi.make_opts(spp=spp, max_depth=4, seed=2, **WAVEFRONT))
    nb, ib = ctx.stats().invalid_samples, ctx.stats().iterations
    assert ia == 1 < ib if w == 64 else 1 < ia <= ib
    assert 0 < na == nb < w * h * spp
    assert np.isfinite(a).all() and np.array_equal(a, b)
    img, = ctx.render_batch([(s, abi.make_opts(spp=spp, max_depth=4, seed=2))])
    assert ctx.stats().invalid_samples == na and np.isfinite(img).all()


def test_contexts_of_one_process_render_side_by_side():
    def job(k, out):
        ctx = api.Context(0)
        s = api.Scene.from_data(ctx, scenes.reference_spheres(200 + k, 150))
        out[k] = [s.render_film(abi.make_opts(spp=spp, max_depth=0, seed=k)) for spp in (1, 4, 9)]
        want = [s.render_film(abi.make_opts(spp=spp, max_depth=0, seed=k, **WAVEFRONT)) for spp in (1, 4, 9)]
        out[k] = all(np.array_equal(a, b) for a, b in zip(out[k], want))
    out = {}
    threads = [threading.Thread(target=job, args=(k, out)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert out == {k: True for k in range(4)}
