"""The work this renderer is timed on, through its Python API.

Every case is one call (or one pair of calls) that a program using the
package makes: plain frames from thumbnail to 1080p and 236 M samples, a
batch of requests, radiance of explicit paths, ray batches, and the guiding
network's inference, training and use in a frame.  The scenes, resolutions
and sample counts are those of the package's own scene generators and tests,
or odd sizes of the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from drawlab_gb300 import abi, api, scenes

_CTX = None
_SKY: dict = {}


def _ctx() -> api.Context:
    """The program's one context: scenes, guides and calls share it."""
    global _CTX
    if _CTX is None:
        _CTX = api.Context(0)
    return _CTX


# ------------------------------------------------------------------- cases

def listed():
    return [
        # a thumbnail for an interactive preview: launches and latency
        dict(name="preview_64", kind="render", scene="cornell", width=64, height=64, spp=1, depth=8, filter="gaussian",
             power=False),
        # the Cornell box at its usual size and sample count
        dict(name="cornell_256", kind="render", scene="cornell", width=256, height=256, spp=16, depth=8,
             filter="gaussian", power=False),
        # all five BSDFs under a sky and an area light, an odd frame size
        dict(name="sky_517x389", kind="render", scene="sky", width=517, height=389, spp=9, depth=8, filter="gaussian",
             power=False),
        # bitmap textures and the box filter
        dict(name="textured_333x251", kind="render", scene="textured", width=333, height=251, spp=12, depth=8,
             filter="box", power=False),
        # the material-sphere frame: 1080p, 64 samples per pixel, 328k triangles
        dict(name="spheres_1080p", kind="render", scene="spheres", width=1920, height=1080, spp=64, depth=16,
             filter="gaussian", power=False),
        # the MIS stress frame with the power-proportional emitter pick
        dict(name="plates_720p", kind="render", scene="plates", width=1280, height=720, spp=256, depth=8,
             filter="gaussian", power=True),
        # requests of uneven size over several scenes in one call
        dict(name="batch_16", kind="batch", requests=16, max_side=512, max_spp=64, triangles=256000),
        # radiance of explicit paths (Integrator::Li), unbounded depth
        dict(name="li_60k", kind="li", width=96, height=64, paths=60007),
        # first hits and shadow queries of a ray batch in host memory
        dict(name="rays_200k", kind="rays", rays=200003),
        # the guiding network: inference on many points, Adam steps on a batch
        dict(name="net_forward", kind="forward", rows=100003),
        dict(name="net_train", kind="learn", records=131072, steps=16),
        # a frame guided by a frozen network
        dict(name="guided_480x270", kind="guided", width=480, height=270, spp=16, depth=12, grid=150),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "batch", "li", "rays", "forward", "learn", "guided"])
    if kind == "render":
        scene = rng.choice(["cornell", "sky", "textured", "spheres", "plates"])
        w, h = _log_int(rng, 32, 1920), _log_int(rng, 32, 1080)
        top = 60e6 if scene in ("spheres", "plates") else 20e6   # samples: below the largest listed frame
        spp = max(1, min(_log_int(rng, 1, 256), int(top / (w * h))))
        return dict(kind=kind, scene=scene, width=w, height=h, spp=spp, depth=rng.choice([0, 5, 8, 16]),
                    filter=rng.choice(["gaussian", "gaussian", "box"]), power=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind=kind, requests=rng.randint(2, 24), max_side=rng.choice([128, 256, 512]),
                    max_spp=rng.choice([4, 16, 64]), triangles=_log_int(rng, 1000, 256000))
    if kind == "li":
        return dict(kind=kind, width=_log_int(rng, 16, 640), height=_log_int(rng, 16, 480),
                    paths=_log_int(rng, 100, 400000))
    if kind == "rays":
        return dict(kind=kind, rays=_log_int(rng, 1, 250000))
    if kind == "forward":
        return dict(kind=kind, rows=_log_int(rng, 1, 400000))
    if kind == "learn":
        return dict(kind=kind, records=_log_int(rng, 64, 200000), steps=rng.randint(1, 32))
    return dict(kind=kind, width=_log_int(rng, 48, 640), height=_log_int(rng, 32, 360), spp=rng.randint(1, 16),
                depth=rng.choice([5, 8, 12]), grid=rng.choice([16, 60, 150]))


# ------------------------------------------------------------------ inputs

def _sky(width, height):
    if (width, height) not in _SKY:
        _SKY[(width, height)] = scenes.sky_envmap(width, height, sun_peak=1.0e4, sun_radius_deg=0.5)
    return _SKY[(width, height)]


def _scene_data(name, width, height, seed):
    if name == "cornell":
        return scenes.cornell(width, height)
    if name == "sky":
        s = scenes.env_spheres(width, height)
        s.lights[-1].env_rgb = _sky(1024, 512)
        return s
    if name == "textured":
        return scenes.textured_cornell(width, height, seed=seed & 0xffff)
    if name == "spheres":
        return scenes.material_spheres(width, height, seed=seed & 0xffff)
    return scenes.mis_plates(width, height)


def _opts(case, seed):
    return abi.make_opts(spp=case["spp"], max_depth=case["depth"], seed=seed,
                         filter=abi.DL_FILTER_BOX if case["filter"] == "box" else abi.DL_FILTER_GAUSSIAN,
                         flags=abi.DL_RENDER_POWER_LIGHT_PICK if case["power"] else 0)


def _network(seed):
    """Parameters of a network after some training: layers of usual scale,
    lobes that vary over positions and normals."""
    r = np.random.default_rng(seed)
    w1 = r.uniform(-1, 1, (64, 144)) * math.sqrt(6 / 144)
    w2 = r.uniform(-1, 1, (64, 64)) * math.sqrt(6 / 64)
    w3 = np.zeros((48, 64))
    w3[:40] = r.uniform(-1, 1, (40, 64)) * 0.5 * math.sqrt(3 / 64)
    b3 = np.zeros(48)
    lobes = r.normal(size=(8, 3))
    b3[:40].reshape(8, 5)[:, :3] = lobes / np.linalg.norm(lobes, axis=1, keepdims=True)
    b3[3:40:5] = r.uniform(0.5, 2.5, 8)
    b = r.uniform(-0.1, 0.1, 128)
    return np.concatenate([w1.ravel(), b[:64], w2.ravel(), b[64:], w3.ravel(), b3]).astype(np.float32)


def _points(r, n):
    """Shading points as the network sees them: position in [0, 1]^3, normal."""
    x = np.empty((n, 6), np.float32)
    x[:, :3] = r.random((n, 3))
    nrm = r.normal(size=(n, 3))
    x[:, 3:] = nrm / np.linalg.norm(nrm, axis=1, keepdims=True)
    return x


def _records(case, seed):
    """Training records: directions around the normal's hemisphere, radiance
    peaked around a position-dependent direction, a few bright ones."""
    r, n = np.random.default_rng(seed), case["records"]
    rec = np.zeros((n, 12), np.float32)
    rec[:, :6] = _points(r, n)
    w = r.normal(size=(n, 3)) + rec[:, 3:6]
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    rec[:, 6:9] = w
    rec[:, 9] = np.maximum((w * rec[:, 3:6]).sum(1), 0.02) / math.pi
    a = math.pi * rec[:, 0]
    mu = np.stack([np.cos(a), np.zeros_like(a), np.sin(a)], 1)
    rec[:, 10] = 0.1 + 5.0 * np.exp(20.0 * ((w * mu).sum(1) - 1.0)) + (r.random(n) < 1e-3) * 200.0
    return rec


def _unit(r, n):
    d = r.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _rays(case, seed):
    """Half camera rays, half bounce rays; and shadow rays towards the lights'
    height, over the material-sphere scene.  n x 8: o, tmin, d, tmax."""
    r, n = np.random.default_rng(seed), case["rays"]
    lo, hi = np.array([-20.0, 0.01, -20.0]), np.array([20.0, 2.5, 20.0])
    close = np.zeros((n, 8), np.float32)
    k = n // 2
    target = r.uniform(lo, hi, (k, 3))
    d = target - np.array([0.0, 9.0, 26.0])
    close[:k, :3] = (0.0, 9.0, 26.0)
    close[:k, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    close[k:, :3] = r.uniform(lo, hi, (n - k, 3))
    close[k:, 4:7] = _unit(r, n - k)
    close[:, 3], close[:, 7] = 1e-4, np.inf
    shadow = np.zeros((n, 8), np.float32)
    o = r.uniform(lo, hi, (n, 3))
    d = r.uniform((-14.0, 8.0, -14.0), (14.0, 12.0, 14.0), (n, 3)) - o
    dist = np.linalg.norm(d, axis=1)
    shadow[:, :3], shadow[:, 4:7] = o, d / dist[:, None]
    shadow[:, 3], shadow[:, 7] = 1e-4, dist - 1e-4
    return close, shadow


def _batch(case, seed):
    """The sizes and sample counts of the requests go by the case; scenes,
    cameras and sample seeds by the seed."""
    sizes, r = np.random.default_rng(case["requests"]), np.random.default_rng(seed)
    tris = sorted({max(1000, case["triangles"] >> k) for k in (0, 2, 4, 8)})
    datas = [scenes.batch_scene(t, (seed + k) & 0xffff, _sky(1024, 512) if k % 2 == 0 else None)
             for k, t in enumerate(tris)]
    items = []
    for k in range(case["requests"]):
        side = case["max_side"] >> int(sizes.integers(0, 3))
        w, h = side + int(sizes.integers(-9, 1)), side + int(sizes.integers(-9, 1))
        spp = max(1, case["max_spp"] >> (2 * int(sizes.integers(0, 2))))
        a = float(r.uniform(0, 2 * math.pi))
        cam = scenes.Camera(width=w, height=h, eye=(16.0 * math.sin(a), 7.0, 16.0 * math.cos(a)),
                            lookat=(0.0, 0.5, 0.0), up=(0.0, 1.0, 0.0), fov=45.0)
        items.append((int(sizes.integers(0, len(datas))), spp, cam, int(r.integers(0, 1 << 31))))
    return datas, items


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    st = dict(kind=kind, ctx=ctx)
    if kind == "render":
        st["scene"] = api.Scene.from_data(ctx, _scene_data(case["scene"], case["width"], case["height"], seed))
        st["opts"] = _opts(case, seed)
    elif kind == "batch":
        datas, items = _batch(case, seed)
        st["scenes"] = [api.Scene.from_data(ctx, d) for d in datas]
        st["items"] = [(st["scenes"][i], abi.make_opts(spp=spp, max_depth=8, seed=s), cam) for i, spp, cam, s in items]
    elif kind == "li":
        st["scene"] = api.Scene.from_data(ctx, scenes.reference_spheres(case["width"], case["height"]))
        st["opts"] = abi.make_opts(max_depth=0, seed=seed)
        r = np.random.default_rng(seed)
        st["xys"] = r.integers(0, (case["width"], case["height"], 64), (case["paths"], 3)).astype(np.int32)
    elif kind == "rays":
        st["scene"] = api.Scene.from_data(ctx, scenes.material_spheres(seed=seed & 0xffff))
        st["close"], st["shadow"] = _rays(case, seed)
    elif kind in ("forward", "learn"):
        st["guide"] = api.Guide(ctx, seed=seed)
        st["guide"].set_params(_network(seed))
        st["steps"] = case.get("steps")
        st["x"] = _points(np.random.default_rng(seed), case["rows"]) if kind == "forward" else _records(case, seed)
    else:
        st["scene"] = api.Scene.from_data(ctx, scenes.guiding_room(case["width"], case["height"], grid=case["grid"],
                                                                   env_width=1024, env_height=512))
        st["guide"] = api.Guide(ctx, seed=seed)
        st["guide"].set_params(_network(seed))
        st["opts"] = abi.make_opts(spp=case["spp"], max_depth=case["depth"], seed=seed)
    return st


# --------------------------------------------------------------------- run

def run(st):
    kind = st["kind"]
    if kind == "render":
        return st["scene"].render(st["opts"])
    if kind == "batch":
        return st["ctx"].render_batch(st["items"])
    if kind == "li":
        return list(st["scene"].li(st["opts"], st["xys"]))
    if kind == "rays":
        return list(st["scene"].trace_closest(st["close"])) + [st["scene"].trace_any(st["shadow"])]
    if kind == "forward":
        return st["guide"].forward(st["x"])
    if kind == "learn":
        return [st["guide"].train(st["x"], st["steps"]), st["guide"].params()]
    return st["scene"].render_guided(st["opts"], st["guide"], train=False)


# -------------------------------------------------------------------- work

_TRIANGLES = dict(cornell=36, sky=1924, textured=1304, spheres=327690, plates=5132)


def work(case):
    """Bytes: what goes in (geometry, rays, records) and comes out, once.
    Operations: per ray about 16 pairs of box tests and 2 triangle tests of
    the tree search, 2.5 rays per sample; the network's multiply-adds."""
    kind = case["kind"]
    ray = 16 * 36 + 2 * 50
    net = 2 * (144 * 64 + 64 * 64 + 64 * 40)
    if kind in ("render", "guided"):
        samples = case["width"] * case["height"] * case["spp"]
        tris = _TRIANGLES[case["scene"]] if kind == "render" else 2 * 2 * case["grid"] ** 2 + 90
        flops = samples * 2.5 * ray
        if kind == "guided":
            flops += samples * 3 * net
        return dict(bytes=case["width"] * case["height"] * 12 + tris * 36, flops=flops)
    if kind == "batch":
        pixels = case["requests"] * case["max_side"] ** 2 * 0.45
        return dict(bytes=pixels * 12 + 1.4 * case["triangles"] * 36, flops=pixels * case["max_spp"] * 0.6 * 2.5 * ray)
    if kind == "li":
        return dict(bytes=case["paths"] * 32 + 1926 * 36, flops=case["paths"] * 3 * ray)
    if kind == "rays":
        return dict(bytes=case["rays"] * (32 + 16 + 32 + 1) + _TRIANGLES["spheres"] * 36, flops=case["rays"] * 2 * ray)
    if kind == "forward":
        return dict(bytes=case["rows"] * 184 + 33472, flops=case["rows"] * net)
    return dict(bytes=case["records"] * 48 + 3 * 66240, flops=case["records"] * case["steps"] * 3 * net)


# ------------------------------------------------------------------- exact

def _layers(p):
    s = np.cumsum([0, 64 * 144, 64, 64 * 64, 64, 48 * 64, 48])
    shapes = [(64, 144), (64,), (64, 64), (64,), (48, 64), (48,)]
    return [p[a:b].reshape(sh) for a, b, sh in zip(s[:-1], s[1:], shapes)]


def _net64(layers, x):
    """The network's 40 outputs in 64 bits: per input (sin, cos)(2^(k-3) pi x)
    for k < 12, two hidden layers of 64 ReLU units."""
    k = 2.0 ** (torch.arange(12, device=x.device, dtype=torch.float64) - 3) * math.pi
    a = x[:, :, None] * k
    e = torch.stack([a.sin(), a.cos()], -1).reshape(len(x), 144)
    w1, b1, w2, b2, w3, b3 = layers
    h = torch.relu(e @ w1.T + b1)
    h = torch.relu(h @ w2.T + b2)
    return (h @ w3.T + b3)[:, :40]


def _loss64(layers, rec):
    o = _net64(layers, rec[:, :6]).reshape(-1, 8, 5)
    m = o[..., :3]
    mu = m / m.norm(dim=-1, keepdim=True)
    kap = o[..., 3].clamp(-3.0, 8.0).exp()
    logc = torch.log(kap / (2 * math.pi * -torch.expm1(-2 * kap)))
    logp = torch.log_softmax(o[..., 4], -1) + logc + kap * ((mu * rec[:, None, 6:9]).sum(-1) - 1)
    ratio = rec[:, 10] / rec[:, 9]
    return -(torch.clamp(ratio / ratio.mean(), max=20.0) * torch.logsumexp(logp, -1)).mean()


def _exact_learn(case, seed, dev):
    p = torch.tensor(_network(seed), dtype=torch.float64, device=dev)
    rec = torch.tensor(_records(case, seed), dtype=torch.float64, device=dev)
    m, v, loss = torch.zeros_like(p), torch.zeros_like(p), torch.zeros(())
    for t in range(1, case["steps"] + 1):
        q = p.clone().requires_grad_(True)
        loss = _loss64(_layers(q), rec)
        loss.backward()
        g = q.grad
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - 2e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return [float(loss.detach()), p]


def _exact_rays(case, seed, dev):
    """t, u, v of every ray's closest hit by testing every triangle."""
    tri = torch.tensor(scenes.material_spheres(seed=seed & 0xffff).triangles(), dtype=torch.float64, device=dev)
    rays = torch.tensor(_rays(case, seed)[0], dtype=torch.float64, device=dev)
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    nv = (n * v0).sum(1)
    # the Moller-Trumbore numerators as products of ray and triangle vectors:
    # u = e2 . ((o - v0) x d), v = -e1 . ((o - v0) x d), t = n . (o - v0), det = -n . d
    c2 = torch.cat([e2, -torch.linalg.cross(e2, v0)], 1).T.contiguous()
    c1 = -torch.cat([e1, -torch.linalg.cross(e1, v0)], 1).T.contiguous()
    nt = n.T.contiguous()
    out = torch.zeros((3, len(rays)), dtype=torch.float64, device=dev)
    step = max(1, int(6e7) // len(tri))
    for a in range(0, len(rays), step):
        o, d = rays[a:a + step, :3], rays[a:a + step, 4:7]
        f = torch.cat([torch.linalg.cross(o, d), d], 1)
        inv = -1.0 / (d @ nt)
        u, v = (f @ c2) * inv, (f @ c1) * inv
        t = (o @ nt - nv) * inv
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 1e-4) & torch.isfinite(inv)
        t = torch.where(ok, t, torch.full((), math.inf, dtype=torch.float64, device=dev))
        best, at = t.min(1)
        hit = torch.isfinite(best)
        rows = torch.arange(len(at), device=dev)
        out[0, a:a + step] = torch.where(hit, best, 0.0)
        out[1, a:a + step] = torch.where(hit, u[rows, at], 0.0)
        out[2, a:a + step] = torch.where(hit, v[rows, at], 0.0)
    return [None, out[0], out[1], out[2], None]


def exact(case, seed):
    """64-bit values of the ray batches and the network.  Frames and path
    radiance have none: which way a path goes hangs on single-precision
    comparisons, so another arithmetic gives other paths."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if case["kind"] == "forward":
        p = torch.tensor(_network(seed), dtype=torch.float64, device=dev)
        x = torch.tensor(_points(np.random.default_rng(seed), case["rows"]), dtype=torch.float64, device=dev)
        return _net64(_layers(p), x)
    if case["kind"] == "learn":
        return _exact_learn(case, seed, dev)
    if case["kind"] == "rays":
        return _exact_rays(case, seed, dev)
    return None
