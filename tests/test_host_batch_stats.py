"""A batch's counters are those of its last frame, whoever waited for it."""


def test_counters_after_a_finish_without_them(host):
    out = host("""
    rp = pk.Pipe(ctx, "raster")
    b = pk.Batch(ctx, [pk.Scene(rp, tri_scene(seed=k)) for k in range(2)])
    for frame in range(1, 8):
        b.run(graph=False)
        if frame % 2:
            assert lib.piko_batch_finish(b.h, None) == 0
        assert b.finish()["covered"] == frame      # (the stub counts the frames it draws)
        assert b.finish()["covered"] == frame
    print("done")
    """)
    assert out == "done\n"
