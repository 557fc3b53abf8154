"""A fresh scene's first frame: device memory is allocated with few calls, each of which
takes several times as long as the frame."""


def test_reyes_allocations(host):
    out = host("""
    yp = pk.Pipe(ctx, "reyes")
    make = lambda: pk.Scene(yp, pk.scenes.sphere_patches(W=320, H=240, seed=1))
    for k in range(40):
        s = make()
        lib.stub_fail_alloc(k, 1)    # the k-th allocation fails, if there is one
        try:
            s.run()
            break
        except pk.PikoError:
            pass
        finally:
            lib.stub_fail_alloc(-1, 0)
    assert 1 <= k <= 2, k            # a block on the device, the counters in pinned memory
    s.finish()
    assert not [x for x in log() if "NULL" in x]
    print("done")
    """)
    assert out == "done\n"
