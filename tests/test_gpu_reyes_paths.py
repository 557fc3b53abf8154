"""Reyes frames that take the less common paths: subtrees that outgrow a CTA of
the split, more micropolygons than get a number each, tables and records that
overflow and grow, and frames queued one behind the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def patches(pk, n, W, H, seed, size):
    """n bicubic patches facing the camera of the sphere workload."""
    sc = pk.scenes.sphere_patches(W=W, H=H)
    g = np.random.Generator(np.random.Philox(seed))
    cps = np.zeros((n, 16, 4), np.float32)
    grid = (np.stack(np.meshgrid(np.arange(4), np.arange(4)), -1).reshape(16, 2) / 3.0 - 0.5) * size
    cps[:, :, :2] = g.uniform(-0.9, 0.9, (n, 1, 2)) * (0.0 if n == 1 else 1.0) + grid
    cps[:, :, 2] = g.uniform(-0.3, 0.3, (n, 16))
    cps[:, :, 3] = 1.0
    sc.patches = cps
    return sc


def draw(pk, ctx, sc, frames=1, **kw):
    pipe = pk.Pipe(ctx, "reyes", **kw)
    s = pk.Scene(pipe, sc)
    try:
        for _ in range(frames):
            s.run()
        fb, depth = s.read()
        return fb, depth, s.stats()
    finally:
        s.close()
        pipe.close()


def same(got, ref):
    fb, depth, st = got
    ofb, odepth, ost = ref
    assert st["prims_kept"] == ost["leaves"] and st["upolys"] == ost["upolys"]
    assert st["covered"] == ost["covered"] and st["split_levels"] == ost["levels"]
    assert np.array_equal(depth.view(np.uint32), odepth.view(np.uint32))
    assert np.array_equal(fb, ofb)


@pytest.mark.parametrize("n,size,thr", [(1, 2.2, 1.5), (5, 1.6, 2.0), (150, 0.5, 2.0), (400, 0.3, 1.5), (1300, 0.1, 2.0)])
def test_split_subtrees(pk, ctx, oracle_mod, n, size, thr):
    sc = patches(pk, n, 640, 480, n, size)
    same(draw(pk, ctx, sc, split_threshold_px=thr, max_splits=18),
         oracle_mod.reyes_frame(sc, threshold=thr, max_splits=18))


def test_more_micropolygons_than_numbers(pk, ctx, oracle_mod):
    sc = pk.scenes.sphere_patches(W=192, H=128)
    same(draw(pk, ctx, sc, frames=2, split_threshold_px=0.5, max_splits=9, dice_grid=32),
         oracle_mod.reyes_frame(sc, threshold=0.5, max_splits=9, grid=32))


@pytest.mark.parametrize("spp,phong", [(1, False), (4, True)])
def test_flat_stack_of_ties(pk, ctx, oracle_mod, spp, phong):
    """Coincident patches: every sample sees many fragments of one depth."""
    sc = patches(pk, 1, 320, 240, 3, 1.2)
    sc.patches[:, :, 2] = 0.25
    sc.patches = np.repeat(sc.patches, 40, axis=0)
    kw = dict(split_threshold_px=12.0, max_splits=10, dice_grid=8)
    fb, depth, st = draw(pk, ctx, sc, frames=3, samples_per_pixel=spp, sample_seed=7, phong=phong, **kw)
    ofb, odepth, ost = oracle_mod.reyes_frame_ms(sc, threshold=12.0, max_splits=10, grid=8, spp=spp, seed=7, phong=phong)
    assert st["covered"] == ost["covered"]
    assert np.array_equal(depth.view(np.uint32), odepth.view(np.uint32))
    assert np.array_equal(fb, ofb)


def test_queued_frames(pk, ctx, oracle_mod):
    """Frames of two scenes queued without a wait: each leaves its counters and
    sample states as the next needs them."""
    scs = [patches(pk, 30, 200, 160, 5, 0.5), pk.scenes.sphere_patches(W=160, H=120)]
    pipe = pk.Pipe(ctx, "reyes")
    scenes = [pk.Scene(pipe, sc) for sc in scs]
    try:
        for s in scenes:
            s.run()
            s.finish()
        for _ in range(20):
            for s in scenes:
                s.run()
        for s, sc in zip(scenes, scs):
            fb, depth = s.read()
            same((fb, depth, s.stats()), oracle_mod.reyes_frame(sc))
    finally:
        for s in scenes:
            s.close()
        pipe.close()
