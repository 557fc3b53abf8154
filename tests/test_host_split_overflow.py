"""A split whose frontier overflows ends at that step, as slots of the frontier were not
written, and the frame is run again with room for all of its patches and for their leaves."""


def test_next_patches(host):
    out = host("""
    fn = lib.stub_next_patches
    fn.restype = ctypes.c_uint32
    for cap in (1 << 16, 100000):
        for count in (0, 1, cap - 1, cap):
            assert fn(count, cap) == count
        for count in (cap + 1, cap + 255, 3 * cap, (1 << 32) - 1):
            assert fn(count, cap) == 0
    print("done")
    """)
    assert out == "done\n"


def test_buffers_grow(host):
    out = host("""
    yp = pk.Pipe(ctx, "reyes")
    for frontier, leaves in [(70000, 1000), (70000, 65000), (300000, 200000), (10, 70000)]:
        s = pk.Scene(yp, pk.scenes.sphere_patches(W=128, H=64, seed=1))
        lib.stub_patches(frontier, leaves)
        s.run()
        s.finish()
        caps = [[int(float(v)) for v in x.split()[4:]] for x in log() if x.startswith("launch reyes_split")]
        assert len(caps) == 2 and caps[0] == [65536, 65536], caps
        assert caps[1][0] >= max(frontier, 65536) and caps[1][1] >= leaves + (frontier if frontier > 65536 else 0), caps
    print("done")
    """)
    assert out == "done\n"
