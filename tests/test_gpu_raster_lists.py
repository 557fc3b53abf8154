"""8x8 tiles with lists of every length around the limits of a pass (two lanes
per entry up to 16 entries, 32 entries a pass, 64 a chunk, several chunks) and
with depths of every kind the nearest-first order has to keep exact: overlapping
planes, equal depths, negative, signed-zero and huge values, wrapping areas."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 8, 9, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 97, 129, 300]


def depths(kind, g, n):
    if kind == "planes":
        return g.uniform(0.05, 0.95, (n, 3))
    if kind == "flat":       # each triangle at one depth, a few depths in all
        return np.repeat(g.choice([0.25, 0.5, 0.75, 1.0], n)[:, None], 3, axis=1)
    if kind == "near":       # differences of a few rounding steps
        return 0.5 + g.integers(-3, 4, (n, 3)) * 2.0 ** -24
    if kind == "signed":
        return g.choice([-0.75, -0.25, -1e-30, -0.0, 0.0, 1e-30, 0.25, 0.75], (n, 3))
    return g.choice([-1e30, -2.0, 0.25, 0.9, 1.5, 1e30], (n, 3))   # "huge"


def payload(kind, n, W, H, seed, size):
    """n counter-clockwise triangles of about `size` pixels around the screen's centre."""
    g = np.random.Generator(np.random.Philox(seed))
    a0 = g.uniform(0, 2 * np.pi, n)
    xyz = np.zeros((n, 9), np.float32)
    z = depths(kind, g, n)
    cx, cy = W / 2 + g.uniform(-6, 6, n), H / 2 + g.uniform(-6, 6, n)
    for k in range(3):
        a = a0 + k * 2 * np.pi / 3 + g.uniform(-0.3, 0.3, n)
        r = size * g.uniform(0.3, 1.0, n)
        xyz[:, 3 * k], xyz[:, 3 * k + 1], xyz[:, 3 * k + 2] = cx + r * np.cos(a), cy + r * np.sin(a), z[:, k]
    icol = (g.integers(0, 1 << 24, (n, 3), dtype=np.uint32) | np.uint32(0xFF000000)).astype(np.uint32)
    return {"W": W, "H": H, "xyz": xyz, "icol": icol}


def check(pk, ctx, oracle_mod, sc, **kw):
    pipe = pk.Pipe(ctx, "raster", tile_px=8, **kw)
    s = pk.Scene(pipe, sc)
    try:
        for _ in range(2):
            s.run()
            fb, depth = s.read()
        st = s.stats()
    finally:
        s.close()
        pipe.close()
    ofb, odepth, ost = oracle_mod.raster_frame(sc["W"], sc["H"], sc["xyz"], sc["icol"])
    assert np.array_equal(depth.view(np.uint32), odepth.view(np.uint32))
    assert np.array_equal(fb, ofb)
    assert st["covered"] == ost["covered"] and st["prims_kept"] == ost["kept"]


@pytest.mark.parametrize("kind", ["planes", "flat", "near", "signed", "huge"])
@pytest.mark.parametrize("size", [3.0, 40.0])
def test_list_lengths(pk, ctx, oracle_mod, kind, size):
    for i, n in enumerate(LENGTHS):
        check(pk, ctx, oracle_mod, payload(kind, n, 64, 72, 100 + i, size))


@pytest.mark.parametrize("chunk", [1, 7, 32, 100, 4096])
def test_chunk_lengths(pk, ctx, oracle_mod, chunk):
    for n in (5, 33, 129, 300):
        check(pk, ctx, oracle_mod, payload("planes", n, 64, 72, n, 40.0), chunk_entries=chunk)


@pytest.mark.parametrize("W,H", [(32, 32), (40, 33), (257, 65), (1021, 767)])
def test_group_sizes(pk, ctx, oracle_mod, W, H):
    """Frames of a few and of many tiles: one to eight tiles per short-list group."""
    sc = pk.scenes.plain_scene(n=4000, W=W, H=H, seed=W, edge_median=0.05)
    xyz, icol = oracle_mod.r1_setup(sc)
    check(pk, ctx, oracle_mod, {"W": W, "H": H, "xyz": xyz, "icol": icol})


def test_wrapping_area(pk, ctx, oracle_mod):
    """Triangles whose doubled area exceeds int32 among small ones."""
    sc = payload("planes", 40, 3200, 3200, 5, 60.0)
    big = np.array([[-200, -200, 0.9, 3400, -200, 0.2, 3400, 3400, 0.6], [-200, -150, 0.3, 3400, 3400, 0.8, -150, 3400, 0.7]],
                   np.float32)
    sc["xyz"] = np.concatenate([big, sc["xyz"]])
    sc["icol"] = np.concatenate([np.full((2, 3), 0xFF3060C0, np.uint32), sc["icol"]])
    check(pk, ctx, oracle_mod, sc)


def spread(kind, n, W, H, seed, size):
    """payload() with the triangles spread over the frame, some of them large."""
    sc = payload(kind, n, W, H, seed, size)
    g = np.random.Generator(np.random.Philox(seed + 1))
    dx, dy = g.uniform(-W / 2, W / 2, n), g.uniform(-H / 2, H / 2, n)
    sc["xyz"][:, 0::3] += dx[:, None].astype(np.float32)
    sc["xyz"][:, 1::3] += dy[:, None].astype(np.float32)
    return sc


@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("chunk", [0, 1, 40, 4096])
def test_bins_of_larger_tiles(pk, ctx, oracle_mod, tile, chunk):
    """16/32-px tiles: a bin's entries gathered from a tile list that other bins
    share, in frames drawn bin by bin and (the large one) quad by quad."""
    cases = [payload("planes", n, 64, 72, n, s) for n in (1, 8, 9, 33, 300) for s in (3.0, 40.0)]
    cases += [payload("signed", 200, 40, 33, 3, 20.0), spread("near", 5000, 333, 257, 4, 6.0)]
    if chunk in (0, 40):
        cases.append(spread("planes", 30000, 1920, 1080, 5, 12.0))
    for sc in cases:
        pipe = pk.Pipe(ctx, "raster", tile_px=tile, chunk_entries=chunk)
        s = pk.Scene(pipe, sc)
        try:
            s.run()
            fb, depth = s.read()
            st = s.stats()
        finally:
            s.close()
            pipe.close()
        ofb, odepth, ost = oracle_mod.raster_frame(sc["W"], sc["H"], sc["xyz"], sc["icol"])
        assert np.array_equal(depth.view(np.uint32), odepth.view(np.uint32))
        assert np.array_equal(fb, ofb)
        assert st["covered"] == ost["covered"]
