"""What bounds the resident kernel: the vertices of one path, not the work of
a warp.  With a library whose limit is 16 vertices, a pass of many short
paths renders what the regular library renders, and a pass with longer paths
ends in DL_ERR_TIMEOUT and leaves the context usable."""
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
s = api.Scene.from_data(ctx, scenes.cornell(512, 512))
t = api.Scene.from_data(ctx, scenes.cornell(100, 64))
short = abi.make_opts(spp=5, max_depth=8, seed=3)
long_ = abi.make_opts(spp=5, max_depth=200, rr_depth=1000, seed=3)
xys = np.array([(x, y, 0) for y in range(64) for x in range(100)], np.int32)
out = dict(film=s.render_film(short), li=t.li(short, xys)[0], batch=ctx.render_batch([(t, short), (s, short)])[1])
if sys.argv[3] == "limited":
    for call in (lambda: s.render(long_), lambda: t.render(long_), lambda: t.li(long_, xys),
                 lambda: ctx.render_batch([(t, long_), (t, long_)])):
        try:
            call()
        except api.DrawlabError as e:
            assert e.status == abi.DL_ERR_TIMEOUT and "did not converge" in str(e), str(e)
        else:
            raise SystemExit("no error")
out["again"] = t.render_film(short)
assert ctx.stats().iterations == 1   # the resident kernel
np.savez(sys.argv[2], **out)
"""


def _run(library, limited, out):
    env = dict(os.environ, DRAWLAB_GB300_LIBRARY=str(library))
    r = subprocess.run([sys.executable, "-c", CHILD, REPO, str(out), "limited" if limited else "regular"], env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return dict(np.load(out))


def test_a_path_not_a_warp_is_bounded(tmp_path):
    from drawlab_gb300 import build
    regular = build.build()
    obj, lib = tmp_path / "resident.cu.o", tmp_path / "libdlgpu_limit.so"
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-DDL_MAX_VERTICES=16", "-c", str(build.CSRC / "resident.cu"),
                    "-o", str(obj)], check=True, timeout=600)
    others = [build.BUILD / (src + ".o") for src in build.CU_SOURCES + build.CPP_SOURCES if src != "resident.cu"]
    subprocess.run([build.NVCC, *build.GENCODE, "-shared", "-o", str(lib), str(obj), *map(str, others),
                    "-cudart", "shared", "-Xcompiler", "-pthread"], check=True, timeout=600)
    a = _run(regular, False, tmp_path / "a.npz")
    b = _run(lib, True, tmp_path / "b.npz")
    assert a.keys() == b.keys()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
