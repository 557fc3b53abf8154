"""Raster frames queued faster than the device draws them: every frame uses the
camera it was prepared with, and the working counters that a frame leaves
behind suit the next frame, whatever its size."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cameras(pk, W, H, n):
    eyes = [(50.0 + 3.0 * k, 8.0, -12.0 + 2.0 * k) for k in range(n)]
    return [pk.camera.view_proj(e, (50.0, 0.0, 40.0), (0.0, 1.0, 0.0), np.radians(60.0), W, H, 0.5, 300.0) for e in eyes]


def forest(pk, n, W, H):
    sc = copy.copy(pk.scenes.forest_scene(W=W, H=H))
    sc.pos, sc.nrm, sc.uv, sc.texture = sc.pos[:, :n], sc.nrm[:, :n], None, None
    return sc


def with_camera(sc, vp):
    sc = copy.copy(sc)
    sc.view_proj = vp
    return sc


@pytest.mark.parametrize("tile", [8, 16, 32])
def test_queued_frames_keep_their_camera(pk, ctx, oracle_mod, tile):
    sc = forest(pk, 20000, 320, 200)
    states = [with_camera(sc, vp) for vp in cameras(pk, sc.W, sc.H, 4)]
    expect = [oracle_mod.raster_scene(s)[:2] for s in states]
    pipe = pk.Pipe(ctx, "raster", tile_px=tile)
    s = pk.Scene(pipe, sc)
    try:
        for st in states:   # the queues settle: a frame that overflows is drawn again with the latest camera
            s.prepare(pk.const_state(st))
            s.run()
            s.finish()
        for last in range(4):
            for k in list(range(4)) * 25 + [last]:   # nothing waits between these
                s.prepare(pk.const_state(states[k]))
                s.run()
            s.prepare(pk.const_state(states[(last + 1) % 4]))   # no frame follows: the image stays
            fb, depth = s.read()
            assert np.array_equal(fb, expect[last][0])
            assert np.array_equal(depth.view(np.uint32), expect[last][1].view(np.uint32))
    finally:
        s.close()
        pipe.close()


def test_queued_batches_keep_their_cameras(pk, ctx, oracle_mod):
    scs = [forest(pk, 9000, 320, 200), forest(pk, 3000, 160, 128), forest(pk, 0, 64, 64)]
    states = [[with_camera(sc, vp) for vp in cameras(pk, sc.W, sc.H, 3)] for sc in scs]
    pipe = pk.Pipe(ctx, "raster", tile_px=8)
    scenes = [pk.Scene(pipe, sc) for sc in scs]
    batch = pk.Batch(ctx, scenes)
    try:
        for k in range(3):   # the queues settle
            for s, st in zip(scenes, states):
                s.prepare(pk.const_state(st[k]))
            batch.run(graph=False)
            batch.finish()
        for last in range(3):
            for k in list(range(3)) * 20 + [last]:
                for s, st in zip(scenes, states):
                    s.prepare(pk.const_state(st[k]))
                batch.run(graph=False)
            for s, st in zip(scenes, states):
                s.prepare(pk.const_state(st[(last + 1) % 3]))
            stats = batch.finish()
            assert stats["prims_kept"] > 0 and stats["status"] == 0
            for s, st in zip(scenes, states):
                fb, depth = s.read()
                ofb, odepth, _ = oracle_mod.raster_scene(st[last])
                assert np.array_equal(fb, ofb)
                assert np.array_equal(depth.view(np.uint32), odepth.view(np.uint32))
    finally:
        batch.close()
        for s in scenes:
            s.close()
        pipe.close()


def test_counters_after_an_overflow_and_an_empty_frame(pk, ctx, oracle_mod):
    """A frame that overflows its lists and is drawn again, graph replays and a
    scene without triangles all leave the counters as the next frame needs them."""
    from helpers import golden, scene_from
    sc = scene_from(pk, golden("raster_guard_giants"))
    xyz, icol = oracle_mod.r1_setup(sc)
    ofb, odepth, ost = oracle_mod.raster_frame(sc.W, sc.H, xyz, icol)
    pipe = pk.Pipe(ctx, "raster", tile_px=8)
    s, empty = pk.Scene(pipe, sc), pk.Scene(pipe, forest(pk, 0, 96, 64))
    batch = pk.Batch(ctx, [s])
    try:
        for _ in range(3):
            empty.run()
            efb, edepth = empty.read()
            assert np.all(efb == 0xFF663313) and np.all(edepth == 1.0)
            s.run()
            s.run()
            fb, depth = s.read()
            st = s.stats()
            assert np.array_equal(fb, ofb) and np.array_equal(depth.view(np.uint32), odepth.view(np.uint32))
            assert st["covered"] == ost["covered"] and st["prims_kept"] == ost["kept"]
            batch.run(graph=True)
            batch.run(graph=True)
            bst = batch.finish()
            assert (bst["covered"], bst["prims_kept"], bst["bin_entries"]) == (st["covered"], st["prims_kept"], st["bin_entries"])
    finally:
        batch.close()
        s.close()
        empty.close()
        pipe.close()
