"""Frames of one scene or batch given to one stream after the other with nothing
waiting in between: each follows the one before, and the frames afterwards equal
those of a scene that never left its stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1].view(np.uint32), b[1].view(np.uint32))


def forest(pk, W, H):
    sc = pk.scenes.forest_scene(W=W, H=H)
    sc.uv = sc.texture = None
    return sc


@pytest.mark.parametrize("kind", ["raster8", "raster32", "reyes", "reyes4"])
def test_scene_frames(pk, ctx, kind):
    import torch
    if kind.startswith("raster"):
        pipe = pk.Pipe(ctx, "raster", tile_px=int(kind[6:]))
        sc = forest(pk, 1277, 715)
    else:
        pipe = pk.Pipe(ctx, "reyes", samples_per_pixel=4 if kind == "reyes4" else 1, phong=kind == "reyes4")
        sc = pk.scenes.sphere_patches(W=640, H=360, seed=4)
    alone, s = pk.Scene(pipe, sc), pk.Scene(pipe, sc)
    try:
        alone.run()
        alone.finish()
        want, stats = alone.read(), alone.stats()
        streams = [torch.cuda.Stream() for _ in range(3)]
        order = [None] + [x.cuda_stream for x in streams]
        s.run()
        s.finish()   # the queues settle
        for turn in range(6):
            for k in range(24):
                s.run(order[(k * (turn + 1)) % 4])
            assert same(s.read(), want), turn
            st = s.stats()
            assert st == stats, turn
        for _ in range(3):
            s.run()
            assert same(s.read(), want)
    finally:
        alone.close()
        s.close()
        pipe.close()


@pytest.mark.parametrize("groups", [1, 2])
@pytest.mark.parametrize("graph", [False, True])
def test_batch_frames(pk, ctx, groups, graph):
    import torch
    pipe = pk.Pipe(ctx, "raster")
    scs = [forest(pk, 640, 360), pk.scenes.plain_scene(n=3000, W=512, H=400, seed=3),
           pk.scenes.plain_scene(n=900, W=200, H=200, seed=5)]
    scenes = [pk.Scene(pipe, sc) for sc in scs]
    tuner = pk.Tuner()
    if groups == 2:
        tuner.set(pk.tune_bucket(640, 360, scs[0].n), 16, 0, 0)
    batch = pk.Batch(ctx, scenes, tuner=tuner)
    try:
        want = []
        for s in scenes:
            s.run()
            want.append(s.read())
        batch.run(graph=graph)
        stats = batch.finish()
        streams = [torch.cuda.Stream() for _ in range(2)]
        order = [None] + [x.cuda_stream for x in streams]
        for turn in range(4):
            for k in range(15):
                batch.run(order[(k * (turn + 1)) % 3], graph=graph)
            assert batch.finish() == stats
            for s, w in zip(scenes, want):
                assert same(s.read(), w), turn
    finally:
        batch.close()
        for s in scenes:
            s.close()
        pipe.close()
