"""How a raster frame's first launch is shaped, for every number of triangles, none
included."""
import pytest


@pytest.mark.parametrize("entry", ["frame", "batch", "noalloc"])
def test_frame_without_triangles(host, entry):
    """The host code is compiled unoptimised here: a division by zero on the way to a
    launch that is not made ends the process."""
    out = host(f"""
    entry = {entry!r}
    pipe = pk.Pipe(ctx, "raster")
    if entry == "noalloc":
        buf = (ctypes.c_uint32 * (64 * 32))()
        p = ctypes.cast(buf, ctypes.c_void_p)
        assert lib.piko_raster_frame_noalloc(p, p, 0, 64, 32, p, p, None) == 0
    else:
        scenes = [pk.Scene(pipe, tri_scene(n=0)) for _ in range(2)]
        if entry == "batch":
            b = pk.Batch(ctx, scenes)
            b.run(graph=True)
            b.finish()
        else:
            scenes[0].run()
            scenes[0].finish()
    lines = log()
    assert any("raster_frag8" in x or "raster_bins" in x for x in lines)
    assert not any("raster_setup" in x for x in lines)
    print("done")
    """)
    assert out == "done\n"


def test_setup_shape(host):
    out = host("""
    fn = lib.stub_setup_shape
    for wave, threads in [(148 * 5, 256), (148 * 8, 128), (7, 32)]:
        full = wave * threads
        for n in [0, 1, 7, 8, 9, 33, 8 * wave - 1, 8 * wave, 8 * wave + 1, 32 * wave + 1, full - 1, full, full + 1, 3 * full + 5,
                  (1 << 32) - 1]:
            batch, blocks = ctypes.c_uint32(), ctypes.c_uint32()
            fn(ctypes.c_uint32(n), ctypes.c_uint32(wave), ctypes.c_uint32(threads), ctypes.byref(batch), ctypes.byref(blocks))
            batch, blocks = batch.value, blocks.value
            assert 8 <= batch <= threads and (batch <= 32 or batch % 32 == 0), (n, batch)
            assert blocks == min(wave, -(-n // batch)), (n, batch, blocks)
            rounds = -(-n // full)    # passes of full CTAs that n triangles take
            assert -(-n // max(blocks * batch, 1)) <= rounds, (n, batch, blocks)
    print("done")
    """)
    assert out == "done\n"
