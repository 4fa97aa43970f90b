"""The resident kernel (passes of few paths in one launch) against the
wavefront: the same paths, the same sums, so films and path radiance are
bit-equal.  A pool size in the options selects the wavefront."""
import numpy as np
import pytest

from drawlab_gb300 import abi, api, scenes

pytestmark = pytest.mark.gpu

PERSPECTIVE = scenes.Camera(width=37, height=23, type=abi.DL_CAMERA_PERSPECTIVE, fov=50.0, far_clip=9.0,
                            transform=scenes.look_at((0.0, 3.0, 9.0), (0.0, 0.5, 0.0), (0.0, 1.0, 0.0)))


@pytest.fixture(scope="module")
def ctx():
    return api.Context(0)


def make(name, w, h):
    if name == "sky":
        return scenes.env_spheres(w, h)
    if name == "spheres":
        return scenes.material_spheres(w, h, num_spheres=8, level=2)
    if name == "perspective":
        s = scenes.reference_spheres(w, h)
        s.camera = PERSPECTIVE
        return s
    if name == "empty":
        return scenes.SceneData("empty", camera=scenes.Camera(width=w, height=h))
    return {"cornell": scenes.cornell, "textured": scenes.textured_cornell, "plates": scenes.mis_plates,
            "refspheres": scenes.reference_spheres}[name](w, h)


# (paths: one; a warp and its neighbours; the edge between 256 and more slots
# a block on 152 SMs, 77824; the edge between the kernel's two shapes, 229376;
# larger passes; the largest, 3 * 2^19)
@pytest.mark.parametrize("name,w,h,spp,depth,flags", [
    ("cornell", 1, 1, 1, 8, 0),
    ("cornell", 31, 1, 1, 0, 0),
    ("cornell", 33, 1, 1, 8, 0),
    ("textured", 304, 256, 1, 8, 0),
    ("textured", 305, 256, 1, 8, 0),
    ("cornell", 448, 512, 1, 8, 0),
    ("cornell", 449, 512, 1, 8, 0),
    ("cornell", 512, 512, 1, 8, 0),
    ("cornell", 513, 512, 1, 8, 0),
    ("cornell", 1024, 768, 2, 4, 0),
    ("sky", 97, 61, 7, 8, 0),
    ("sky", 300, 301, 5, 0, abi.DL_RENDER_POWER_LIGHT_PICK),
    ("textured", 83, 47, 9, 8, 0),
    ("plates", 131, 77, 3, 8, abi.DL_RENDER_POWER_LIGHT_PICK),
    ("refspheres", 96, 64, 3, 0, abi.DL_RENDER_FIX_POINT_LIGHT),
    ("refspheres", 250, 130, 16, 0, 0),
    ("spheres", 160, 90, 4, 16, 0),
    ("perspective", 37, 23, 5, 6, 0),
    ("sky", 64, 33, 3, 8, abi.DL_RENDER_NORMALS),
    ("empty", 40, 30, 2, 8, 0),
])
def test_resident_film_equals_wavefront(ctx, name, w, h, spp, depth, flags):
    s = api.Scene.from_data(ctx, make(name, w, h))
    a = s.render_film(abi.make_opts(spp=spp, max_depth=depth, seed=5, flags=flags))
    sa = ctx.stats()
    b = s.render_film(abi.make_opts(spp=spp, max_depth=depth, seed=5, flags=flags, max_paths_in_flight=1 << 16))
    sb = ctx.stats()
    assert sa.iterations == 1 and sb.iterations > 1   # the two paths ran
    assert np.array_equal(a, b)
    assert (sa.camera_rays, sa.extension_rays, sa.shadow_rays) == (sb.camera_rays, sb.extension_rays, sb.shadow_rays)


@pytest.mark.parametrize("n", [1, 32, 1000, 300000])
def test_resident_paths_equal_wavefront(ctx, n):
    s = api.Scene.from_data(ctx, scenes.reference_spheres(96, 64))
    xys = np.random.default_rng(n).integers(0, (96, 64, 50), (n, 3)).astype(np.int32)
    a = s.li(abi.make_opts(seed=9), xys)
    assert ctx.stats().iterations == 1
    b = s.li(abi.make_opts(seed=9, max_paths_in_flight=4096), xys)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_resident_batch_equals_single_renders(ctx):
    names = ["cornell", "sky", "plates", "textured", "refspheres"]
    made = [api.Scene.from_data(ctx, make(n, 40 + 7 * k, 31 + 5 * k)) for k, n in enumerate(names)]
    items = [(s, abi.make_opts(spp=3 + k, max_depth=6, seed=k)) for k, s in enumerate(made)]
    imgs = ctx.render_batch(items)
    assert ctx.stats().iterations == 1
    for (s, o), img in zip(items, imgs):
        o.max_paths_in_flight = 8192
        assert np.array_equal(img, s.render(o))


# more than 3 * 2^19 paths: the wavefront, whose last paths the resident kernel
# takes over (unbounded and bounded depth, paths that all end in the first
# graph launch); a pool size keeps the wavefront to the end
@pytest.mark.parametrize("name,w,h,spp,depth", [
    ("cornell", 1025, 768, 2, 4),
    ("refspheres", 640, 480, 7, 0),
    ("sky", 1024, 700, 3, 0),
    ("textured", 801, 663, 5, 12),
    ("spheres", 1201, 449, 4, 3),
    ("empty", 1450, 1449, 1, 0),
])
def test_finished_wavefront_equals_wavefront(ctx, name, w, h, spp, depth):
    s = api.Scene.from_data(ctx, make(name, w, h))
    a = s.render_film(abi.make_opts(spp=spp, max_depth=depth, seed=6))
    sa = ctx.stats()
    b = s.render_film(abi.make_opts(spp=spp, max_depth=depth, seed=6, max_paths_in_flight=1 << 24))
    sb = ctx.stats()
    assert 1 < sa.iterations <= sb.iterations and (depth or name == "empty" or sa.iterations < sb.iterations)
    assert np.array_equal(a, b)
    assert (sa.camera_rays, sa.extension_rays, sa.shadow_rays) == (sb.camera_rays, sb.extension_rays, sb.shadow_rays)


def test_finished_wavefront_paths_and_batch(ctx):
    s = api.Scene.from_data(ctx, scenes.reference_spheres(96, 64))
    n = (1 << 21) + 77
    xys = np.random.default_rng(3).integers(0, (96, 64, 400), (n, 3)).astype(np.int32)
    a = s.li(abi.make_opts(seed=9), xys)
    b = s.li(abi.make_opts(seed=9, max_paths_in_flight=1 << 24), xys)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    made = [api.Scene.from_data(ctx, make(m, 700, 500)) for m in ("refspheres", "sky")]
    items = [(m, abi.make_opts(spp=5, max_depth=0, seed=k)) for k, m in enumerate(made)]
    imgs = ctx.render_batch(items)
    for (m, o), img in zip(items, imgs):
        o.max_paths_in_flight = 1 << 24
        assert np.array_equal(img, m.render(o))
