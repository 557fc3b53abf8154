"""Arrays that read() and getData() hand out: never one that the caller still
holds, in any form, and the depth buffer filled in place or by copy alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_held_arrays_stay(pk, ctx):
    pipe = pk.Pipe(ctx, "raster")
    a, b = pk.scenes.plain_scene(n=500, W=96, H=64, seed=1), pk.scenes.plain_scene(n=500, W=96, H=64, seed=2)
    s = pk.Scene(pipe, a)
    try:
        s.run()
        fb, depth = s.read()
        want_fb, want_depth = fb.copy(), depth.copy()
        view, flat = fb[10:20, ::2], depth.reshape(-1).view(np.uint32)
        held = [fb, depth]
        del fb, depth
        s.upload(b)
        for _ in range(5):
            s.run()
            other_fb, other_depth = s.read()
            assert not np.array_equal(other_fb, want_fb)
            assert all(o is not h for o in (other_fb, other_depth) for h in held)
        assert np.array_equal(held[0], want_fb) and np.array_equal(held[1], want_depth)
        del held, other_fb, other_depth
        for _ in range(3):      # only views are left
            s.run()
            s.read()
        assert np.array_equal(view, want_fb[10:20, ::2]) and np.array_equal(flat, want_depth.reshape(-1).view(np.uint32))
    finally:
        s.close()
        pipe.close()


@pytest.mark.parametrize("form", ["exact", "longer", "strided", "float64"])
def test_depth_buffer_forms(pk, ctx, form):
    W, H = 96, 64
    sc = pk.scenes.plain_scene(n=800, W=W, H=H, seed=3)
    ms = pk.MutableState(W, H)
    if form == "longer":
        ms.zBuffer = np.full(W * H + 100, 7.0, np.float32)
    elif form == "strided":
        ms.zBuffer = np.full(2 * W * H, 7.0, np.float32)[::2]
    elif form == "float64":
        ms.zBuffer = np.full(W * H, 7.0)
    pipe = pk.RasterPipe(ctx)
    pipe.allocate(pk.ConstantState(W, H), ms, sc)
    for _ in range(2):
        pipe.prepare()
        pipe.run_single()
        data = pipe.pikoScreen.getData()
    fb, depth = pipe._scene.read()
    assert np.array_equal(data.reshape(H, W), fb)
    assert np.array_equal(np.asarray(ms.zBuffer[: W * H], np.float32).view(np.uint32), depth.reshape(-1).view(np.uint32))
    assert form != "longer" or np.all(ms.zBuffer[W * H:] == 7.0)
    pipe.destroy()
