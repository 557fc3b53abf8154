"""Sizes at the edges of the groups that raster_setup and reyes_dice work in: scenes
of a few triangles to a few CTAs' worth in one launch sequence, and dice grids
around the number of leaves whose points share a group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1, 7, 8, 9), (31, 32, 33, 127), (128, 129, 255, 256, 257), (5000, 1, 40000)])
@pytest.mark.parametrize("tile", [8, 16])
def test_setup_of_several_scenes(pk, ctx, oracle_mod, counts, tile):
    pipe = pk.Pipe(ctx, "raster", tile_px=tile)
    src = [pk.scenes.plain_scene(n=n, W=200 + i, H=120 + 8 * i, seed=n, edge_median=0.08) for i, n in enumerate(counts)]
    scenes = [pk.Scene(pipe, s) for s in src]
    batch = pk.Batch(ctx, scenes)
    try:
        batch.run()
        batch.finish()
        for sc, s in zip(src, scenes):
            fb, depth = s.read()
            ofb, odepth, _ = oracle_mod.raster_frame(sc.W, sc.H, *oracle_mod.r1_setup(sc))
            assert np.array_equal(fb, ofb)
            assert np.array_equal(depth.view(np.uint32), odepth.view(np.uint32))
    finally:
        batch.close()
        for s in scenes:
            s.close()
        pipe.close()


@pytest.mark.parametrize("grid", [1, 2, 8, 15, 16, 17, 31, 32])
def test_dice_groups(pk, ctx, oracle_mod, grid):
    sc = pk.scenes.sphere_patches(W=320, H=240)
    pipe = pk.Pipe(ctx, "reyes", split_threshold_px=24.0, max_splits=8, dice_grid=grid)
    s = pk.Scene(pipe, sc)
    try:
        s.run()
        fb, depth = s.read()
        st = s.stats()
    finally:
        s.close()
        pipe.close()
    ofb, odepth, ost = oracle_mod.reyes_frame(sc, threshold=24.0, max_splits=8, grid=grid)
    assert st["upolys"] == ost["upolys"] and st["covered"] == ost["covered"]
    assert np.array_equal(fb, ofb)
    assert np.array_equal(depth.view(np.uint32), odepth.view(np.uint32))
