"""What a replayed frame draws with: the cameras of the last frame that was enqueued
without the graph, the same for batches of one and of several scenes, for one-scene
groups among larger ones, and for captures of the caller's own."""
import pytest

MAKE = """
rp = pk.Pipe(ctx, "raster")
small = lambda k: pk.Scene(rp, tri_scene(seed=k))
large = lambda k: pk.Scene(rp, tri_scene(W=320, H=300, n=9000, seed=k))

def shown():      # the cameras of the frames drawn since, in the order of their groups
    return [[float(c) for c in x.split()[4:]] for x in log() if x.startswith(("launch raster_frag8", "launch raster_bins"))]

def aim(scenes, x):
    for i, s in enumerate(scenes):
        s.prepare(camera(x + i))
"""


@pytest.mark.parametrize("scenes,tuned,groups", [
    ("[small(1)]", False, [[0]]), ("[small(1), small(2)]", False, [[0, 1]]),
    ("[small(1), large(2)]", True, [[0], [1]]), ("[small(1), large(2), small(3)]", True, [[0, 2], [1]])])
def test_batch(host, scenes, tuned, groups):
    out = host(MAKE + f"""
scenes = {scenes}
tuner = pk.Tuner()
tuner.set(pk.tune_bucket(320, 300, 9000), 16, 0, 0)
b = pk.Batch(ctx, scenes, tuner=tuner if {tuned} else None)
want = lambda x: [[x + i for i in g] for g in {groups}]
aim(scenes, 10.0)
b.run(graph=True)
b.finish()
log()
for step in range(3):
    aim(scenes, 20.0 + 10 * step)
    b.run(graph=True)                 # (a replay takes no notice of prepare())
    assert shown() == want(10.0 + 10 * step), step
    b.run(graph=False)
    assert shown() == want(20.0 + 10 * step), step
    aim(scenes, 7.0)
    for _ in range(2):
        b.run(graph=True)
        lines = log()
        assert not [x for x in lines if "memset" in x]
        got = [[float(c) for c in x.split()[4:]] for x in lines if x.startswith(("launch raster_frag8", "launch raster_bins"))]
        assert got == want(20.0 + 10 * step), (step, got)
    b.finish()
print("done")
""")
    assert out == "done\n"


@pytest.mark.parametrize("n,graph", [(0, False), (1, False), (2, False), (1, True), (2, True)])
def test_callers_capture(host, n, graph):
    """n = 0: a scene's own frame; else a batch of n scenes, its launches captured (graph:
    the batch has a graph of its own, whose run is captured)."""
    out = host(MAKE + f"""
scenes = [small(k) for k in range(max({n}, 1))]
f = pk.Batch(ctx, scenes) if {n} else scenes[0]
go = (lambda s=None, graph=False: f.run(s, graph=graph)) if {n} else f.run
want = lambda x: [[x + i for i in range(len(scenes))]]
aim(scenes, 10.0)
go()
f.finish()
a = lib.stub_stream()
if {graph}:
    go(graph=True)
aim(scenes, 20.0)
lib.stub_begin_capture(a)
if {graph}:
    go(a, graph=True)
else:
    go(a)
g = lib.stub_end_capture(a)
log()
lib.stub_replay(g, a)
lines = log()
assert "memset" in lines[0], lines                  # (a replay starts from cleared counters)
got = [[float(c) for c in x.split()[4:]] for x in lines if x.startswith(("launch raster_frag8", "launch raster_bins"))]
assert got == want(10.0 if {graph} else 20.0), got  # (a run of the graph takes no notice of prepare())
for x in (30.0, 40.0):
    aim(scenes, x)
    go()
    f.finish()
    assert shown() == want(x)
    aim(scenes, 5.0)
    for _ in range(2):
        lib.stub_replay(g, a)
        got = shown()
        assert got == want(x), (x, got)
    if {graph}:
        for _ in range(2):
            go(graph=True)
            lines = log()
            assert "memset" in [y for y in lines if y.startswith(("memset", "launch"))][0], lines
        f.finish()
print("done")
""")
    assert out == "done\n"
