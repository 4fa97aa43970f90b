"""The bounds-checked build over both programs a render may run: the
wavefront for single renders, batches and explicit paths (a pool size given),
the resident kernel in each of its shapes, and a wavefront that the resident
kernel finishes.  No violation, and images bit-equal to the regular
library's."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from drawlab_gb300 import abi, api, scenes
ctx = api.Context(0)
out = {}
def made(name, w, h):
    f = dict(cornell=scenes.cornell, sky=scenes.env_spheres, plates=scenes.mis_plates,
             textured=scenes.textured_cornell, refspheres=scenes.reference_spheres)[name]
    return api.Scene.from_data(ctx, f(w, h))
def run(key, resident, call):
    out[key] = call()
    it = ctx.stats().iterations
    assert it == 1 if resident else it > 1, (key, it)
small = {k: made(k, 48, 33) for k in ("cornell", "sky", "plates", "textured", "refspheres")}
for pool in (0, 512, 1 << 16):
    for name, s in small.items():
        o = abi.make_opts(spp=5, max_depth=8, seed=3, max_paths_in_flight=pool)
        run("%s_%d" % (name, pool), pool == 0, lambda: s.render_film(o))
    o = abi.make_opts(spp=3, max_depth=8, seed=4, flags=abi.DL_RENDER_POWER_LIGHT_PICK, max_paths_in_flight=pool)
    run("power_%d" % pool, pool == 0, lambda: small["sky"].render_film(o))
    o = abi.make_opts(max_depth=0, seed=5, max_paths_in_flight=pool)
    xys = np.random.default_rng(6).integers(0, (48, 33, 9), (5001, 3)).astype(np.int32)
    run("li_%d" % pool, pool == 0, lambda: small["refspheres"].li(o, xys)[0])
    items = [(s, abi.make_opts(spp=2 + k, max_depth=6, seed=k, max_paths_in_flight=pool))
             for k, s in enumerate(small.values())]
    run("batch_%d" % pool, pool == 0, lambda: np.concatenate([im.ravel() for im in ctx.render_batch(items)]))
for w in (300, 512):     # the resident kernel's shapes for more paths
    s = made("sky", w, w)
    run("wide_sky_%d" % w, True, lambda: s.render_film(abi.make_opts(spp=1, max_depth=8, seed=7)))
    run("wide_skies_%d" % w, True, lambda: ctx.render_batch([(s, abi.make_opts(spp=1, max_depth=8, seed=8))])[0])
s = made("refspheres", 640, 480)   # a finished wavefront
o = abi.make_opts(spp=6, max_depth=0, seed=9)
run("finished", False, lambda: s.render_film(o))
run("finished_batch", False, lambda: ctx.render_batch([(s, o)])[0])
np.savez(sys.argv[2], **out)
"""


def _run(library, out):
    env = dict(os.environ, DRAWLAB_GB300_LIBRARY=str(library))
    r = subprocess.run([sys.executable, "-c", CHILD, REPO, str(out)], env=env, capture_output=True, text=True,
                       timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return dict(np.load(out))


def test_both_programs_render_without_violations(tmp_path):
    from drawlab_gb300 import build
    a = _run(build.build(checked=True), tmp_path / "checked.npz")
    b = _run(build.build(), tmp_path / "regular.npz")
    assert a.keys() == b.keys() and len(a) == 30
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
