"""Contexts on two devices of one process: what a kernel needs raised on its
device (the limit of dynamic shared memory) is raised on each of them, so the
second device's launches go through like the first's."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import fake_cudart  # noqa: E402

CODE = r"""
def use(device):
    ctx = api.Context(device)
    one = api.Scene.from_data(ctx, scenes.cornell(300, 300))
    few, many, more = (api.Scene.from_data(ctx, scenes.cornell(w, w)) for w in (64, 512, 1280))
    opts = lambda **k: abi.make_opts(spp=1, max_depth=4, **k)
    for s in (few, one, many, more):       # the resident kernel's shapes; the wavefront and its end
        s.render(opts())
    for s in (few, one, many, more):       # the same for batches
        ctx.render_batch([(s, opts())])
    g = api.Guide(ctx, seed=1)
    g.forward(np.zeros((300, 6), np.float32))
    g.train(np.ones((300, 12), np.float32), 2)
    few.render_guided(opts(), g, train=False)
    ran = {l.split()[2] for l in log() if l.startswith("launch %d " % device)}
    refused = [l for l in log() if l.startswith("refused")]
    assert not refused, refused
    return ran

first, second = use(0), use(1)
assert first == second
for kernel in ("k_resident", "k_material", "k_guide_infer", "k_guide_train", "k_film_gather"):
    print(kernel, sum(kernel in k for k in first))
"""


def test_both_devices_take_every_launch(tmp_path):
    out = fake_cudart.run(CODE, tmp_path)
    ran = dict((k, int(v)) for k, v in (line.split() for line in out.splitlines()))
    assert ran["k_resident"] == 8            # three shapes and the wavefront's end, single and batch
    assert ran["k_guide_infer"] == ran["k_guide_train"] == 1 and ran["k_film_gather"] == 2
    assert ran["k_material"] >= 13           # five types, single and batch, and three guided ones
