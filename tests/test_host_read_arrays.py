"""The memory of read()'s images: never one that the caller still holds, in any form and
whatever an interpreter's reference counts are; a bounded number kept for the next."""


def test_held_images(host):
    out = host("""
    sys.getrefcount = lambda o: 3       # (counts of objects differ from one interpreter to the next)
    s = pk.Scene(pk.Pipe(ctx, "raster"), tri_scene())
    address = lambda a: a.__array_interface__["data"][0]
    def draw():
        s.run()
        return s.read()
    held = [draw() for _ in range(5)]
    assert len({address(a) for pair in held for a in pair}) == 10
    fb, depth = held[0]
    assert fb.shape == depth.shape == (64, 96) and fb.dtype == np.uint32 and depth.dtype == np.float32
    assert fb.flags.writeable and fb.flags.c_contiguous and fb.flags.aligned
    views = [held[1][0][10:20, ::2], held[1][1].reshape(-1).view(np.uint32), memoryview(held[2][0]), held[2][1].T]
    kept = {address(a) for pair in held[:3] for a in pair}
    del held[1:], fb, depth             # views hold two more pairs
    for _ in range(6):
        a, b = draw()
        assert not {address(a), address(b)} & kept
    del a, b
    assert [len(v) for v in s._free.values()] == [2, 2]
    before = draw()
    at = [address(a) for a in before]
    del before
    assert [address(a) for a in draw()] == at       # let go of: taken again
    again = draw()
    s.close()
    again[0][:] = 7                                 # outlives the scene
    del s
    assert (again[0] == 7).all() and again[1].sum() is not None
    print("done")
    """)
    assert out == "done\n"
