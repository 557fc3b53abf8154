"""A read-back that fails leaves the caller's depth buffer as it was."""
import pytest


@pytest.mark.parametrize("form", ["exact", "longer", "strided"])
def test_depth_buffer_after_a_failure(host, form):
    out = host(f"""
    W, H = 96, 64
    ms = pk.MutableState(W, H)
    if {form!r} == "longer":
        ms.zBuffer = np.ones(W * H + 100, np.float32)
    if {form!r} == "strided":
        ms.zBuffer = np.ones(2 * W * H, np.float32)[::2]
    ms.zBuffer[:] = 7.0
    pipe = pk.RasterPipe(ctx)
    pipe.allocate(pk.ConstantState(W, H), ms, tri_scene(W=W, H=H))
    pipe.prepare()
    lib.stub_overflow(1)             # the lists are too short, and there is no memory for longer ones
    def fails(call):
        try:
            call()
        except pk.PikoError as e:
            assert e.status == 2, e  # PIKO_ERR_OOM
            return
        assert False
    pipe._scene.run()
    lib.stub_fail_alloc(0, 2)
    fails(pipe._scene.finish)        # (run_single() is the two)
    fails(pipe.pikoScreen.getData)
    assert (ms.zBuffer == 7.0).all()
    log()
    pipe.pikoScreen.getData()        # with memory for them the frame is drawn again
    assert [x.split()[1] for x in log() if x.startswith("launch")].count("raster_frag8") == 1
    assert (ms.zBuffer[: W * H] == 0.0).all() and (ms.zBuffer[W * H:] == 7.0).all()     # (the stub draws zeros)
    print("done")
    """)
    assert out == "done\n"
