"""Launch shapes set by the caller are the ones renders use, and images do not
depend on them."""
import numpy as np
import pytest

from drawlab_gb300 import abi, api, scenes

pytestmark = pytest.mark.gpu


def test_iterations_per_graph_set_by_the_caller_are_kept():
    # more paths than the resident kernel takes alone, few vertices each: the
    # render ends with the first graph launch after its last vertex
    ctx = api.Context(0)
    s = api.Scene.from_data(ctx, scenes.cornell(1300, 1250))
    opts = abi.make_opts(spp=1, max_depth=2, seed=1)
    s.render(opts)
    assert ctx.stats().iterations in (2, 4)   # none set: looked at after every two
    t = ctx.get_tune()
    assert t.iterations_per_graph == 8
    for k in (8, 6, 4, 2, 8):
        t.iterations_per_graph = k
        ctx.set_tune(t)
        assert ctx.get_tune().iterations_per_graph == k
        s.render(opts)
        it = ctx.stats().iterations
        assert it == k or (k == 2 and it == 4)


def test_autotune_times_what_renders_run():
    # unbounded paths through glass: a render looks for its last paths and
    # finishes them in one launch, and so does a trial (here the last one, of
    # eight iterations a graph)
    ctx = api.Context(0)
    s = api.Scene.from_data(ctx, scenes.reference_spheres(640, 480))
    opts = abi.make_opts(spp=16, max_depth=0, seed=2)
    t, _ = ctx.autotune([(s, opts)], trial_spp=2)
    assert ctx.stats().iterations == 8
    s.render(opts)
    assert ctx.stats().iterations < 150   # (232 to the end, at an eighth of the samples)


@pytest.mark.parametrize("threads", [64, 128, 256])
def test_launch_shapes_render_the_same_images(threads):
    # a pool size keeps small frames on the wavefront, which has a launch shape
    ctx = api.Context(0)
    made = [api.Scene.from_data(ctx, f(48, 40)) for f in (scenes.cornell, scenes.env_spheres, scenes.reference_spheres)]
    items = [(s, abi.make_opts(spp=4 + k, max_depth=6, seed=k, max_paths_in_flight=8192)) for k, s in enumerate(made)]
    ref = ctx.render_batch([(s, abi.make_opts(spp=4 + k, max_depth=6, seed=k)) for k, s in enumerate(made)])
    for iterations, trav, shade in ((2, 1, 1), (4, 4, 8), (6, 16, 64), (8, 8, 16)):
        ctx.set_tune(abi.dl_tune_params(paths_in_flight=1 << 20, traverse_ctas_per_sm=trav, shade_ctas_per_sm=shade,
                                        iterations_per_graph=iterations, shade_threads=threads))
        for (s, o), img, want in zip(items, ctx.render_batch(items), ref):
            assert np.array_equal(img, want) and np.array_equal(s.render(o), want)
            assert ctx.stats().iterations > 1
