"""The film gather's two tile sizes against a splat of the same samples (their
radiance and film positions from dl_li) in 64 bits."""
import numpy as np
import pytest

from drawlab_gb300 import abi, api, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return api.Context(0)


def filter_table(filt):
    """The reference's 32-entry filter table (rfilter.cpp, block.cpp)."""
    radius = 0.5 if filt == abi.DL_FILTER_BOX else 2.0
    x = np.float32(radius) * np.arange(32, dtype=np.float32) / np.float32(32)
    if filt == abi.DL_FILTER_BOX:
        t = np.ones(32, np.float32)
    else:
        t = np.maximum(0, np.exp(np.float32(-2) * x * x) - np.exp(np.float32(-8))).astype(np.float32)
    return np.append(t, np.float32(0)), np.float32(32 / radius), 0 if filt == abi.DL_FILTER_BOX else 2


def splat(L, pos, w, h, filt):
    table, lookup, b = filter_table(filt)
    film = np.zeros((h + 2 * b, w + 2 * b, 4))
    p = (pos - np.float32(0.5)) + np.float32(b)
    ix, iy = pos[:, 0].astype(int) + b, pos[:, 1].astype(int) + b
    v = np.concatenate([L.astype(np.float64), np.ones((len(L), 1))], 1)
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            cx, cy = ix + dx, iy + dy
            wx = table[np.minimum((np.abs(cx.astype(np.float32) - p[:, 0]) * lookup).astype(int), 32)]
            wy = table[np.minimum((np.abs(cy.astype(np.float32) - p[:, 1]) * lookup).astype(int), 32)]
            ok = (cx >= 0) & (cx < film.shape[1]) & (cy >= 0) & (cy < film.shape[0])
            np.add.at(film, (cy[ok], cx[ok]), (wx.astype(np.float64) * wy)[ok, None] * v[ok])
    return film


# film sizes: one pixel; one tile of 16 and a column or row more; ragged small
# frames; frames on both sides of three tiles of 32 for four of 152 SMs (112
# and 114 tiles); frames with more of them, whole and ragged
@pytest.mark.parametrize("filt", [abi.DL_FILTER_GAUSSIAN, abi.DL_FILTER_BOX])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 3), (12, 12, 2), (13, 12, 2), (16, 17, 2), (61, 35, 5), (444, 252, 2), (604, 188, 2),
                                     (508, 316, 1),
                                     (509, 320, 2), (640, 479, 1)])
def test_film_equals_a_splat_of_its_samples(ctx, w, h, spp, filt):
    s = api.Scene.from_data(ctx, scenes.cornell(w, h))
    o = abi.make_opts(spp=spp, max_depth=3, seed=8, filter=filt)
    film = s.render_film(o)
    y, x, k = np.mgrid[0:h, 0:w, 0:spp]
    L, pos = s.li(o, np.stack([x.ravel(), y.ravel(), k.ravel()], 1))
    want = splat(L, pos, w, h, filt)
    # sums of at most 25 spp non-negative terms, each with a few roundings
    assert np.abs(film - want).max() <= 25 * spp * 2.0 ** -23 * want.max()
    assert np.all(np.abs(film - want) <= 25 * spp * 2.0 ** -23 * want + 1e-30)
