"""Replayed frames after the camera moved (test_host_replay.py states the rule): the
batch's own graph and a capture of the caller's, whose one scene is read from a table
by the kernels of several scenes, draw the images that a run with that camera draws."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1].view(np.uint32), b[1].view(np.uint32))


def moved(pk, sc, x):
    cs = pk.const_state(sc)
    cs.view_proj[12] = cs.view_proj[12] + x
    return cs


@pytest.mark.parametrize("tile", [8, 16])
@pytest.mark.parametrize("form", ["scene", "batch1", "batch2", "batch1_capture", "batch2_graph_capture"])
def test_moved_camera(pk, ctx, tile, form):
    import torch
    scs = [pk.scenes.plain_scene(n=3000, W=333, H=250, seed=3), pk.scenes.plain_scene(n=500, W=200, H=200, seed=5)]
    scs = scs[: 2 if form.startswith("batch2") else 1]
    pipe = pk.Pipe(ctx, "raster", tile_px=tile)
    plain, scenes = [pk.Scene(pipe, sc) for sc in scs], [pk.Scene(pipe, sc) for sc in scs]
    batch = None if form == "scene" else pk.Batch(ctx, scenes)
    try:
        want = {}
        for x in (0.0, 0.1, -0.2):
            for k, sc in enumerate(scs):
                plain[k].prepare(moved(pk, sc, x))
                plain[k].run()
                want[x, k] = plain[k].read()
        assert not same(want[0.0, 0], want[0.1, 0])

        def aim(x):
            for s, sc in zip(scenes, scs):
                s.prepare(moved(pk, sc, x))

        def check(x):
            for k, s in enumerate(scenes):
                assert same(s.read(), want[x, k]), (x, k)

        def run():
            if batch:
                batch.run(graph=False)
                batch.finish()
            else:
                scenes[0].run()
                scenes[0].finish()

        aim(0.0)
        run()
        if form == "scene" or "capture" in form:
            st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
            own = "graph" in form       # the batch has a graph of its own by then
            if own:
                batch.run(graph=True)
                batch.finish()
            with torch.cuda.graph(g, stream=st):
                if batch:
                    batch.run(st.cuda_stream, graph=own)
                else:
                    scenes[0].run(st.cuda_stream)

            def replay():
                g.replay()
                torch.cuda.synchronize()
        else:
            def replay():
                batch.run(graph=True)
                batch.finish()
        replay()
        check(0.0)
        for x in (0.1, -0.2):
            aim(x)
            run()
            check(x)
            aim(0.0)
            for _ in range(2):
                replay()
                check(x)
        if form == "scene" or "capture" in form:
            del g
    finally:
        if batch:
            batch.close()
        for s in scenes + plain:
            s.close()
        pipe.close()
