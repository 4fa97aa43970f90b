"""A call that fails after its first kernel or copy on the caller's arrays was
launched waits for it before it returns: the caller may free the arrays."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import fake_cudart  # noqa: E402

CODE = r"""
ctx = api.Context(0)
s = api.Scene.from_data(ctx, scenes.cornell(32, 32))
rays = np.ones((100, 8), np.float32)
for failing, call in (("k_split_hits", s.trace_closest), ("k_copy_bytes", s.trace_any)):
    fake.fake_fail_kernel(failing.encode(), 0)
    fake.fake_clear_log()
    try:
        call(rays)
    except api.DrawlabError:
        pass
    else:
        raise SystemExit("no error")
    calls = log()
    assert any(c.startswith("launch") and "k_trace_rays" in c for c in calls)
    assert calls[-1] == "wait", calls
    fake.fake_fail_kernel(b"", 0)
    call(rays)
# a batch whose second image fails: the first one's copy is on its way
fake.fake_fail_kernel(b"k_resolve", 1)
fake.fake_clear_log()
try:
    ctx.render_batch([(s, abi.make_opts(spp=1))] * 2)
except api.DrawlabError:
    pass
else:
    raise SystemExit("no error")
calls = log()
assert "copy" in calls and calls[-1] == "wait", calls
print("ok")
"""


def test_failed_calls_wait_for_their_kernels(tmp_path):
    assert fake_cudart.run(CODE, tmp_path).strip() == "ok"
