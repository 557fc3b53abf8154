"""Frames of one scene or one batch on several streams: the working counters that a
frame leaves for the next one are never changed by two frames at once, whichever
streams they are given and whether anything waits in between."""
import pytest

MAKE = """
rp, yp = pk.Pipe(ctx, "raster"), pk.Pipe(ctx, "reyes")
def make(kind):
    if kind == "raster":
        return pk.Scene(rp, tri_scene())
    if kind == "reyes":
        return pk.Scene(yp, pk.scenes.sphere_patches(W=128, H=64, seed=1))
    tuner = pk.Tuner()    # two groups: two launch sequences side by side
    tuner.set(pk.tune_bucket(256, 200, 900), 8, 0, 32)
    tuner.set(pk.tune_bucket(320, 300, 9000), 16, 0, 0)
    scenes = [pk.Scene(rp, tri_scene(W=256, H=200, n=900)), pk.Scene(rp, tri_scene(W=320, H=300, n=9000, seed=2))]
    make.keep = scenes, tuner
    return pk.Batch(ctx, scenes, tuner=tuner)
"""


@pytest.mark.parametrize("kind,graph", [("raster", None), ("reyes", None), ("batch", False), ("batch", True)])
def test_frames_follow_one_another(host, kind, graph):
    out = host(MAKE + f"""
f = make({kind!r})
go = f.run if {graph!r} is None else (lambda s=None: f.run(s, graph={graph!r}))
a, b = lib.stub_stream(), lib.stub_stream()
for s in [None, a, b, a, a, None, b, None, None, a]:   # nothing waits between these
    go(s)
f.finish()
for s in [a, None, b]:
    go(s)
    f.finish()
lines = log()
assert sum("raster_setup" in x or "reyes_split" in x for x in lines) >= 13
bad = [x for x in lines if "RACE" in x or "NULL" in x]
assert not bad, bad
print("done")
""")
    assert out == "done\n"


@pytest.mark.parametrize("kind", ["raster", "reyes", "batch"])
def test_stream_that_is_gone(host, kind):
    """A caller's stream may be destroyed behind a frame that nothing waited for; the next
    frame, on another stream, still follows that frame and uses the handle no more."""
    out = host(MAKE + f"""
f = make({kind!r})
b = lib.stub_stream()
for _ in range(3):
    a = lib.stub_stream()
    f.run(a)
    lib.stub_destroy_stream(a)
    f.run(b)
f.finish()
bad = [x for x in log() if "RACE" in x or "GONE" in x]
assert not bad, bad
print("done")
""")
    assert out == "done\n"


@pytest.mark.parametrize("kind", ["raster", "reyes"])
def test_captured_frames_clear_their_counters(host, kind):
    """Nothing orders the replays of a caller's own capture with other frames, so a
    captured frame, and every frame of that scene from then on, starts from cleared
    counters: whatever a replay at the wrong time leaves is gone one frame later."""
    out = host(MAKE + f"""
f = make({kind!r})
f.run()
f.finish()
a = lib.stub_stream()
log()
f.run()
f.finish()
assert not [x for x in log() if "memset" in x]     # a frame of a scene that was never captured
lib.stub_begin_capture(a)
f.run(a)
g = lib.stub_end_capture(a)
assert not [x for x in log() if "launch" in x]
first = {{"raster": "raster_setup", "reyes": "reyes_split"}}[{kind!r}]
for replay in (lambda: lib.stub_replay(g, a), lambda: f.run(a), lambda: lib.stub_replay(g, a)):
    replay()
    lines = [x.split(" stream")[0] for x in log() if "memset" in x or "launch" in x]
    assert "memset" in lines[: lines.index("launch " + first)], lines
print("done")
""")
    assert out == "done\n"
