"""Allocations that fail: the call or request reports it, no buffer is used that is not
there, and the next call with memory available draws its frame."""


def test_frames(host):
    """Each allocation of a frame in turn, device and pinned memory alike, in a fresh
    scene and in one that grew; a frame after the failure uses no null buffer, also when
    it needs less than the one that failed."""
    out = host("""
    rp, yp = pk.Pipe(ctx, "raster"), pk.Pipe(ctx, "reyes")
    small, big = tri_scene(), tri_scene(W=256, H=200, n=900)
    kinds = {
        "raster": lambda: [pk.Scene(rp, big)],
        "reyes": lambda: [pk.Scene(yp, pk.scenes.sphere_patches(W=128, H=64, seed=1))],
        "batch": lambda: [pk.Scene(rp, small), pk.Scene(rp, big)],
    }
    for kind, make in kinds.items():
        failed = 0
        for k in range(40):
            scenes = make()
            frame = pk.Batch(ctx, scenes) if kind == "batch" else scenes[0]
            go = (lambda: frame.run(graph=False)) if kind == "batch" else frame.run
            lib.stub_fail_alloc(k, 1)
            try:
                go()
                ok = True
            except pk.PikoError as e:
                assert e.status == 2, e     # PIKO_ERR_OOM
                ok = False
                failed += 1
            lib.stub_fail_alloc(-1, 0)
            frame.finish()
            go()
            frame.finish()
            lines = log()
            assert not [x for x in lines if "NULL" in x], (kind, k, [x for x in lines if "NULL" in x])
            if ok:
                break
        assert ok and failed >= (2 if kind == "reyes" else 8), (kind, failed)
    print("done")
    """)
    assert out == "done\n"


def test_server(host):
    """The same through the served form, whose lanes share their buffers between requests
    of all sizes: the request that met the failure fails (or waits for its output slot),
    the worker lives, and smaller and equal requests after it are drawn."""
    out = host("""
    rp, yp = pk.Pipe(ctx, "raster"), pk.Pipe(ctx, "reyes")
    scenes = {
        "raster": [pk.Scene(rp, tri_scene()), pk.Scene(rp, tri_scene(W=256, H=200, n=9000))],
        "reyes": [pk.Scene(yp, pk.scenes.sphere_patches(W=128, H=64, seed=1)),
                  pk.Scene(yp, pk.scenes.sphere_patches(W=256, H=128, seed=2))],
    }
    def status(server, s):
        rid = server.submit(s, pk.const_state(), keep=True)
        try:
            server.wait(rid)
            server.read(rid, s.W, s.H)
            return 0
        except pk.PikoError as e:
            return e.status
    for kind, (small, big) in scenes.items():
        for warm in (False, True):
            failed = 0
            for k in range(30):
                server = pk.Server(ctx, lanes=1, max_batch=4, max_slots=8, max_pixels=256 * 200)
                if warm:
                    assert status(server, small) == 0
                lib.stub_fail_alloc(k, 1)
                st = status(server, big)
                lib.stub_fail_alloc(-1, 0)
                assert st in (0, 2), (kind, k, st)
                failed += st == 2
                assert status(server, small) == 0 and status(server, big) == 0, (kind, warm, k)
                server.close()
                bad = [x for x in log() if "NULL" in x]
                assert not bad, (kind, warm, k, bad)
            assert failed >= 2, (kind, warm, failed)   # (a warm Reyes lane lacks only its sample buffers)
    print("done")
    """)
    assert out == "done\n"
