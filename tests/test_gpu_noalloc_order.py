"""piko_raster_frame_noalloc takes every frame of up to 2^20 queue entries, in whatever
order its triangles come: its lists cannot grow, and the warps that meet all the large
triangles must not run out of room while the others' stays empty."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = H = 1024
LIMIT = 1 << 20
OK, OVERFLOW = 0, 3
TRI = np.array([10.0, 10.0, 0.5, 262.0, 12.0, 0.5, 14.0, 260.0, 0.5], np.float32)   # 16 x 16 box tiles of 16 px


def payload(places):
    """65,536 triangles, degenerate but for those at `places`, each at a depth of its own."""
    xyz = np.zeros((1 << 16, 9), np.float32)
    xyz[places] = TRI
    xyz[places, 2::3] = np.linspace(0.9, 0.1, len(places), dtype=np.float32)[:, None]
    icol = np.full((1 << 16, 3), 0xFF102030, np.uint32) + np.arange(1 << 16, dtype=np.uint32)[:, None]
    return {"W": W, "H": H, "xyz": xyz, "icol": icol}


def regular(pk, ctx, sc):
    pipe = pk.Pipe(ctx, "raster", tile_px=16)
    s = pk.Scene(pipe, sc)
    try:
        s.run()
        fb, depth = s.read()
        return fb, depth, s.stats()["bin_entries"]
    finally:
        s.close()
        pipe.close()


def noalloc(pk, sc):
    import torch
    d_xyz, d_icol = torch.from_numpy(sc["xyz"]).cuda(), torch.from_numpy(sc["icol"].view(np.int32)).cuda()
    d_fb = torch.full((H, W), 7, dtype=torch.int32, device="cuda")
    d_z = torch.full((H, W), -3.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (d_xyz, d_icol, d_fb, d_z)]
    st = pk.load_library().piko_raster_frame_noalloc(ptr[0], ptr[1], len(sc["xyz"]), W, H, ptr[2], ptr[3], None)
    return st, d_fb.cpu().numpy().view(np.uint32), d_z.cpu().numpy()


@pytest.mark.parametrize("group", [1, 64, 96, 128, 1 << 16])
def test_up_to_the_limit(pk, ctx, group):
    """The large triangles in runs of `group`, 16 runs apart (of one run: at the front), just
    below the limit, where nearly every slot is needed, and just above it."""
    each = regular(pk, ctx, payload(np.array([5])))[2]
    assert each > 100
    most = LIMIT // each
    i = np.arange(1 << 16)
    order = np.concatenate([i[(i // group) % 16 == 0], i[(i // group) % 16 != 0]])
    for k in (3000, most):
        sc = payload(np.sort(order[:k]))
        fb, depth, entries = regular(pk, ctx, sc)
        assert entries == k * each
        st, nfb, nz = noalloc(pk, sc)
        assert st == OK, k
        assert np.array_equal(nfb, fb) and np.array_equal(nz.view(np.uint32), depth.view(np.uint32))
    assert noalloc(pk, payload(np.sort(order[: most + 1])))[0] == OVERFLOW
