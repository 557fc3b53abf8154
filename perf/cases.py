"""Performance cases of piko-public_b200: frames drawn through its public entry
points (Scene, Batch, RasterPipe, upload/read), over the range of sizes that the
package's own workloads, tests and benchmark use.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program holds before a frame (contexts, pipes, scenes; everything from
the seed), run() is one frame, work() its algorithmic bytes, and exact() the
depth buffer in 64-bit arithmetic from plain torch.  Colours are whole numbers
(RGBA8 words).

A case's "form" is how a program drives the frame:

  frame   Scene.prepare + Scene.run + Scene.finish: one frame with its camera
          state, waited for (an interactive loop)
  stream  the same without the wait: the device image goes to a consumer on the
          program's stream (Reyes frames)
  graph   Batch.run over one scene, a replayed CUDA graph (the benchmark's form)
  batch   Batch.run over many scenes, one replayed CUDA graph
  app     RasterPipe.prepare / run_single / pikoScreen.getData, the calls of the
          reference's own application loop; the image comes back to the host
  upload  Scene.upload from pinned host memory, Scene.run, Scene.read
"""
import math

import numpy as np
import torch

import piko_loader

pk = piko_loader.load()

_shared = {}


def _context():
    if "ctx" not in _shared:
        _shared["ctx"] = pk.Context(device=0)
        _shared["stream"] = torch.cuda.Stream()
    return _shared["ctx"]


def _stream():
    _context()
    return _shared["stream"].cuda_stream


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one small interactive frame: the launches and the wait are most of it
        _raster("small_frame", "frame", "plain", 1000, 256, 256),
        # the reference's application loop on its own pre-transformed payload, at
        # the size its plain CPU case has; image and depth read back every frame
        _raster("app_4096_512", "app", "wtri", 4096, 512, 512),
        # few large triangles reaching into the guard band, at an odd size: deep
        # tile lists and much overdraw
        _raster("giants_odd", "graph", "plain", 1500, 1021, 767, edge=0.4, reach=1.4),
        # the largest scene of the batched mix: many small triangles
        _raster("plain_200k_1080p", "graph", "plain", 200000, 1920, 1080),
        # the scene-scale frame: 174,000 textured triangles, perspective camera
        _raster("forest_1080p", "graph", "forest", 174000, 1920, 1080, textured=True),
        # the same forest from a moving camera, Gouraud, packed float3 input, ragged size
        _raster("forest_odd_packed", "frame", "forest", 174000, 1277, 715, packed=True),
        # world-space raster_wtri payload through 16-px tiles
        _raster("world_16px", "frame", "world", 61200, 800, 600, tile=16),
        # scenes of many sizes drawn by one launch sequence
        {"name": "mix24", "form": "batch", "kind": "mix", "scenes": 24, "mix": 3, "tile": 8},
        # Reyes with fixed 16x16 grids, four jittered samples and Phong shading
        _reyes("reyes_4spp_720p", "stream", 1280, 720, thr=16.0, splits=10, grid=16, spp=4, phong=True),
        # Reyes with the reference's constants (4 px, extent-derived grids, one sample)
        _reyes("reyes_ref_768p", "frame", 1024, 768),
        # a small Reyes frame: the levels of the split and the launches count
        _reyes("reyes_small", "frame", 320, 240, thr=16.0, splits=10, grid=16),
        # new geometry every frame: the packed forest from pinned host memory to
        # the device, drawn, colour and depth read back
        _raster("forest_upload", "upload", "forest", 174000, 1920, 1080, textured=True, packed=True),
    ]


def _raster(name, form, kind, n, W, H, tile=8, edge=0.02, reach=1.0, textured=False, packed=False):
    return {"name": name, "form": form, "kind": kind, "n": n, "W": W, "H": H, "tile": tile, "edge": edge,
            "reach": reach, "textured": textured, "packed": packed}


def _reyes(name, form, W, H, thr=0.0, splits=0, grid=0, spp=1, phong=False):
    return {"name": name, "form": form, "kind": "reyes", "W": W, "H": H, "thr": thr, "splits": splits, "grid": grid,
            "spp": spp, "phong": phong}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    W, H = _log_int(rng, 200, 1920), _log_int(rng, 200, 1080)
    what = rng.choice(["plain", "plain", "wtri", "giants", "forest", "forest", "world", "reyes", "reyes", "mix"])
    form = rng.choice(["frame", "graph"])
    tile = rng.choice([8, 8, 8, 16, 32])
    if what == "reyes":
        spp = rng.choice([1, 4])
        if rng.random() < 0.5:   # extent-derived grids, the reference's threshold and about it
            c = _reyes("", "frame", min(W, 1280), min(H, 768), thr=rng.choice([0.0, 4.0, 6.5]), spp=spp,
                       phong=rng.random() < 0.5)
        else:
            c = _reyes("", "stream", min(W, 1280), min(H, 768), thr=rng.uniform(12.0, 24.0), splits=rng.choice([10, 12]),
                       grid=rng.choice([8, 12, 16]), spp=spp, phong=rng.random() < 0.5)
    elif what == "mix":
        c = {"form": "batch", "kind": "mix", "scenes": rng.randint(4, 20), "mix": rng.randint(10, 10000), "tile": tile}
    elif what == "forest":
        packed = rng.random() < 0.5
        c = _raster("", "upload" if packed and rng.random() < 0.3 else form, "forest", 174000, W, H, tile=tile,
                    textured=rng.random() < 0.5, packed=packed)
    elif what == "world":
        c = _raster("", form, "world", 102 * _log_int(rng, 20, 1700), W, H, tile=tile)
    elif what == "giants":
        c = _raster("", form, "plain", _log_int(rng, 100, 1500), W, H, tile=tile, edge=rng.uniform(0.1, 0.4),
                    reach=rng.uniform(0.5, 1.4))
    elif what == "wtri":
        c = _raster("", rng.choice(["app", "frame"]), "wtri", _log_int(rng, 1000, 60000), W, H, tile=tile,
                    edge=rng.uniform(0.01, 0.05))
    else:
        c = _raster("", form, "plain", _log_int(rng, 1000, 200000), W, H, tile=tile, edge=rng.uniform(0.01, 0.03),
                    packed=rng.random() < 0.3)
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return np.random.Generator(np.random.Philox(int(seed)))


def _forest(seed, n, W, H, textured):
    """The forest workload (scenes.forest_scene's sizes and distributions),
    built without a loop over its objects: cones of 51 side and 51 base
    triangles and, at full size, 300 quads on a 100x100 ground grid."""
    g = _rng(seed)
    segs = 51
    full = n == pk.scenes.FOREST_TRIS
    quads = pk.scenes.FOREST_QUADS if full else 0
    cones = (n - 2 * quads) // (2 * segs)
    m = cones + quads
    x, z = g.uniform(0.0, 100.0, (2, m))
    h = g.lognormal(0.0, 0.6, m)
    yaw = g.uniform(0.0, 2.0 * np.pi, m)

    def pt(px, py, pz):
        return np.stack(np.broadcast_arrays(px, py, pz), axis=-1)

    cx, cz, ch = x[:cones, None], z[:cones, None], h[:cones, None]
    r = 0.35 * ch
    a0 = yaw[:cones, None] + np.arange(segs) * (2.0 * np.pi / segs)
    a1 = yaw[:cones, None] + np.arange(1, segs + 1) * (2.0 * np.pi / segs)
    am = 0.5 * (a0 + a1)
    b0, b1 = pt(cx + r * np.cos(a0), 0.0, cz + r * np.sin(a0)), pt(cx + r * np.cos(a1), 0.0, cz + r * np.sin(a1))
    apex, centre = pt(cx + 0.0 * a0, ch, cz), pt(cx + 0.0 * a0, 0.0, cz)

    def side(a):
        return pt(np.cos(a) * ch, r, np.sin(a) * ch)

    down = pt(0.0 * a0, -1.0, 0.0)
    k = np.broadcast_to(np.arange(segs) / segs, a0.shape)
    uv_side = [np.stack([k + 1.0 / segs, 0 * k], -1), np.stack([k, 0 * k], -1), np.stack([k + 0.5 / segs, 0 * k + 1], -1)]
    uv_base = [np.stack([0 * k + 0.5, 0 * k + 0.5], -1), np.stack([0.5 + 0.5 * np.cos(a0), 0.5 + 0.5 * np.sin(a0)], -1),
               np.stack([0.5 + 0.5 * np.cos(a1), 0.5 + 0.5 * np.sin(a1)], -1)]

    def join(sides, bases):
        # per cone and segment: a side triangle, then a base triangle
        return [np.stack([s, b], axis=2).reshape(-1, s.shape[-1]) for s, b in zip(sides, bases)]

    P = join([b1, b0, apex], [centre, b0, b1])
    N = join([side(a1), side(a0), side(am)], [down, down, down])
    U = join(uv_side, uv_base)
    if quads:
        qx, qz, qh, qy = x[cones:], z[cones:], h[cones:], yaw[cones:]
        w = 0.4 * qh
        d = pt(np.cos(qy) * w, 0.0, np.sin(qy) * w)
        o = pt(qx, 0.0, qz)
        up = pt(0.0 * qh, qh, 0.0)
        p0, p1, p2, p3 = o - d, o + d, o + d + up, o - d + up
        qn = pt(-np.sin(qy), 0.0, np.cos(qy))
        t = np.broadcast_to
        one = [t(np.array(c, np.float64), (quads, 2)) for c in ((0, 0), (1, 0), (1, 1), (0, 1))]
        for s, (a, b) in enumerate(((p0, p0), (p1, p2), (p2, p3))):
            P[s] = np.concatenate([P[s], np.stack([a, b], 1).reshape(-1, 3)])
            N[s] = np.concatenate([N[s], np.repeat(qn, 2, axis=0)])
        for s, (a, b) in enumerate(((0, 0), (1, 2), (2, 3))):
            U[s] = np.concatenate([U[s], np.stack([one[a], one[b]], 1).reshape(-1, 2)])
    pos = np.ones((3, n, 4), np.float32)
    nrm = np.zeros((3, n, 4), np.float32)
    pos[:, :, :3] = np.stack(P)
    N = np.stack(N)
    nrm[:, :, :3] = N / np.linalg.norm(N, axis=2, keepdims=True)
    eye = np.array([50.0 + g.uniform(-4.0, 4.0), 8.0 + g.uniform(-1.0, 1.0), -12.0])
    vp = pk.camera.view_proj(eye, (50.0, 0.0, 40.0), (0.0, 1.0, 0.0), np.radians(60.0), W, H, 0.5, 300.0)
    uv = tex = None
    if textured:
        uv = np.ascontiguousarray(np.stack(U), np.float32)
        tex = g.integers(0, 256, (512, 512, 4), dtype=np.uint8)
        tex[:, :, 3] = 255
    return pk.scenes.RasterScene(W=W, H=H, pos=pos, nrm=nrm, col=None, view_proj=vp, light_mode=pk.scenes.LIGHT_EYE,
                                 eye=eye.astype(np.float32), uv=uv, texture=tex)


def _wtri(case, seed):
    """The pre-transformed payload: screen positions and lit vertex colours."""
    sc = pk.scenes.plain_scene(n=case["n"], W=case["W"], H=case["H"], seed=seed, edge_median=case["edge"],
                               xy_range=case["reach"])
    xyz = np.empty((case["n"], 9), np.float32)
    for k in range(3):
        xyz[:, 3 * k] = (sc.pos[k, :, 0] + np.float32(1.0)) * np.float32(0.5 * case["W"])
        xyz[:, 3 * k + 1] = (sc.pos[k, :, 1] + np.float32(1.0)) * np.float32(0.5 * case["H"])
        xyz[:, 3 * k + 2] = sc.pos[k, :, 2]
    rgb = (sc.col[:, :, :3] * np.float32(255.0)).astype(np.uint32)
    icol = np.uint32(0xFF000000) | (rgb[..., 2] << 16) | (rgb[..., 1] << 8) | rgb[..., 0]
    return xyz, np.ascontiguousarray(icol.T)


def _world(case, seed):
    sc = _forest(seed, case["n"], case["W"], case["H"], False)
    xyz = np.ascontiguousarray(sc.pos[:, :, :3].transpose(1, 0, 2).reshape(case["n"], 9))
    return {"W": case["W"], "H": case["H"], "xyz_world": xyz, "view_proj": sc.view_proj}


def _mix_sizes(case):
    """Triangle counts (log-uniform, 1K to 200K) and resolutions of a mix."""
    g = _rng(10000 + case["mix"])
    res = [(256, 256), (512, 512), (1280, 720), (1920, 1080)]
    return [(int(round(math.exp(g.uniform(math.log(1000.0), math.log(200000.0))))),) + res[int(g.integers(0, len(res)))]
            for _ in range(case["scenes"])]


def _reyes_scene(case, seed):
    return pk.scenes.sphere_patches(seed=seed, W=case["W"], H=case["H"])


def _raster_scene(case, seed):
    if case["kind"] == "forest":
        return _forest(seed, case["n"], case["W"], case["H"], case["textured"])
    if case["kind"] == "world":
        return _world(case, seed)
    if case["kind"] == "wtri":
        xyz, icol = _wtri(case, seed)
        return {"W": case["W"], "H": case["H"], "xyz": xyz, "icol": icol}
    return pk.scenes.plain_scene(n=case["n"], W=case["W"], H=case["H"], seed=seed, edge_median=case["edge"],
                                 xy_range=case["reach"])


# ------------------------------------------------------------------ state
class _DeviceImage:
    """A scene's device buffer seen by torch (no copy)."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


class _Resources:
    """The handles behind a state; the device memory goes back with the last
    user of it, an image included."""

    def __init__(self):
        self.scenes, self.pipe, self.batch, self.app = [], None, None, None

    def __del__(self):
        try:
            torch.cuda.synchronize()
            if self.batch is not None:
                self.batch.close()
            for s in self.scenes:
                s.close()
            if self.app is not None:
                self.app.destroy()
            if self.pipe is not None:
                self.pipe.close()
        except Exception:
            pass


class _State:
    """What a program keeps between frames."""

    def __init__(self, form):
        self.form, self.res, self.out = form, _Resources(), []

    def add(self, scene, packed=False):
        s = pk.Scene(self.res.pipe, scene, packed=packed)
        self.res.scenes.append(s)
        fb, depth = s.device_buffers()
        self.out.append((torch.as_tensor(_DeviceImage(self.res, fb, (s.H, s.W), "<i4"), device="cuda"),
                         torch.as_tensor(_DeviceImage(self.res, depth, (s.H, s.W), "<f4"), device="cuda")))


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    t.copy_(torch.from_numpy(a))
    return t.numpy()


def prepare(case, seed):
    ctx = _context()
    form, st = case["form"], _State(case["form"])
    if form == "app":
        xyz, icol = _wtri(case, seed)
        tris = np.zeros(case["n"], pk.raster_wtri)
        tris["id"] = np.arange(case["n"])
        for k in range(3):
            tris[f"worldPos{k}"] = xyz[:, 3 * k:3 * k + 3]
            tris[f"icol{k}"] = icol[:, k]
        st.mutable = pk.MutableState(case["W"], case["H"])
        st.res.app = pk.RasterPipe(ctx, tile_px=case["tile"])
        st.res.app.allocate(pk.ConstantState(case["W"], case["H"]), st.mutable, tris, case["n"])
        return st
    if case["kind"] == "reyes":
        st.res.pipe = pk.Pipe(ctx, "reyes", split_threshold_px=case["thr"], max_splits=case["splits"],
                              dice_grid=case["grid"], samples_per_pixel=case["spp"], sample_seed=7, phong=case["phong"])
        scenes = [_reyes_scene(case, seed)]
    else:
        st.res.pipe = pk.Pipe(ctx, "raster", tile_px=case["tile"])
        if case["kind"] == "mix":
            scenes = [pk.scenes.plain_scene(n=n, W=W, H=H, seed=1000 * (seed + 1) + i)
                      for i, (n, W, H) in enumerate(_mix_sizes(case))]
        else:
            scenes = [_raster_scene(case, seed)]
    packed = case.get("packed", False)
    for sc in scenes:
        st.add(sc, packed)
    if form in ("graph", "batch"):
        st.res.batch = pk.Batch(ctx, st.res.scenes)
        st.res.batch.run(_stream(), graph=True)
        st.res.batch.finish()
        return st
    if form in ("frame", "stream"):
        sc = scenes[0]
        st.const = pk.const_state(view_proj=sc.get("view_proj")) if isinstance(sc, dict) else pk.const_state(sc)
    if form == "stream":
        # the first frame settles the queue sizes
        st.res.scenes[0].run(_stream())
        st.res.scenes[0].finish()
    if form == "upload":
        sc = scenes[0]
        sc.pos = _pinned(np.ascontiguousarray(sc.pos[..., :3])) if packed else _pinned(sc.pos)
        sc.nrm = _pinned(np.ascontiguousarray(sc.nrm[..., :3])) if packed else _pinned(sc.nrm)
        if sc.uv is not None:
            sc.uv, sc.texture = _pinned(sc.uv), _pinned(sc.texture)
        st.desc, st.keep = pk.runtime.scene_desc(sc, packed=packed)
        st.fb = _pinned(np.zeros((sc.H, sc.W), np.int32))
        st.depth = _pinned(np.zeros((sc.H, sc.W), np.float32))
    return st


# ------------------------------------------------------------------ one frame
def run(st):
    form = st.form
    if form in ("frame", "stream"):
        s = st.res.scenes[0]
        s.prepare(st.const)
        s.run(_stream())
        if form == "frame":
            s.finish()
    elif form in ("graph", "batch"):
        st.res.batch.run(_stream(), graph=True)
    elif form == "app":
        st.res.app.prepare()
        st.res.app.run_single()
        return st.res.app.pikoScreen.getData().view(np.int32), st.mutable.zBuffer
    elif form == "upload":
        s = st.res.scenes[0]
        s.upload(st.desc, _stream())
        s.run(_stream())
        s.read(st.fb, st.depth)
        return st.fb, st.depth
    return st.out


# ------------------------------------------------------------------ work
def _scene_bytes(kind, n, W, H, textured=False, packed=False):
    """Each input read once, colour and depth written once."""
    if kind == "wtri":
        per = 48
    elif kind == "world":
        per = 36
    else:
        per = (72 if packed else 96) + (48 if kind in ("plain", "mix") else 0) + (24 if textured else 0)
    return n * per + W * H * 8 + (512 * 512 * 4 if textured else 0)


def work(case):
    if case["kind"] == "mix":
        b = sum(_scene_bytes("mix", n, W, H) for n, W, H in _mix_sizes(case))
    elif case["kind"] == "reyes":
        b = 32 * 16 * 16 + case["W"] * case["H"] * 8
    else:
        b = _scene_bytes(case["kind"], case["n"], case["W"], case["H"], case["textured"], case["packed"])
    return {"bytes": b, "flops": 0}


# ------------------------------------------------------------------ 64 bits
_CHUNK = 1 << 24   # candidate samples per step


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _expand(w, h):
    """Groups of consecutive items with at most _CHUNK cells in all: yields
    (item index, x, y) of every cell of their w x h rectangles."""
    cnt = w * h
    cum = torch.cumsum(cnt, 0)
    n, first = cnt.numel(), 0
    while first < n:
        base = int(cum[first - 1]) if first else 0
        last = max(first + 1, int(torch.searchsorted(cum, torch.tensor(base + _CHUNK, device=cum.device), right=True)))
        c = cnt[first:last]
        i = torch.repeat_interleave(torch.arange(first, last, device=w.device), c)
        q = torch.arange(i.numel(), device=w.device) - (torch.cumsum(c, 0) - c)[i - first]
        yield i, q % w[i], q // w[i]
        first = last


def _raster_depth(W, H, screen):
    """Depth buffer of triangles with screen-space vertices [N, 3, 3] (float64):
    28.4 positions by truncation, back-face, guard-band and between-rows culls,
    edge functions at the pixel centres, the nearest depth below 1."""
    X, Y = (screen[..., 0] * 16.0).trunc().to(torch.int64), (screen[..., 1] * 16.0).trunc().to(torch.int64)
    Z = screen[..., 2]
    guard = 225 * 16
    keep = (Y[:, 2] - Y[:, 0]) * (X[:, 1] - X[:, 0]) - (X[:, 2] - X[:, 0]) * (Y[:, 1] - Y[:, 0]) > 0
    keep &= ((X >= -guard) & (X < W * 16 + guard) & (Y >= -guard) & (Y < H * 16 + guard)).all(1)
    keep &= ((Y.amin(1) - 8) >> 4) != ((Y.amax(1) - 8) >> 4)
    X, Y, Z = X[keep], Y[keep], Z[keep]
    xe, ye = W // 8 * 8, H // 8 * 8     # whole 8x8 bins only
    x0, x1 = ((X.amin(1) + 7) >> 4).clamp(min=0), ((X.amax(1) - 8) >> 4).clamp(max=xe - 1)
    y0, y1 = ((Y.amin(1) + 7) >> 4).clamp(min=0), ((Y.amax(1) - 8) >> 4).clamp(max=ye - 1)
    some = (x1 >= x0) & (y1 >= y0)
    X, Y, Z, x0, x1, y0, y1 = (v[some] for v in (X, Y, Z, x0, x1, y0, y1))
    depth = torch.ones(W * H, dtype=torch.float64, device=X.device)
    dX, dY = X.roll(-1, 1) - X, Y.roll(-1, 1) - Y
    area = (Y[:, 2] - Y[:, 0]) * (X[:, 1] - X[:, 0]) - (X[:, 2] - X[:, 0]) * (Y[:, 1] - Y[:, 0])
    if X.shape[0]:
        for i, x, y in _expand(x1 - x0 + 1, y1 - y0 + 1):
            x, y = x + x0[i], y + y0[i]
            e = [((y * 16 + 8) - Y[i, k]) * dX[i, k] - ((x * 16 + 8) - X[i, k]) * dY[i, k] for k in range(3)]
            cov = (e[0] >= 0) & (e[1] >= 0) & (e[2] >= 0)
            i, p, e1, e2 = i[cov], (y * W + x)[cov], e[1][cov], e[2][cov]
            a = area[i].double()
            z = Z[i, 2] + e1 / a * (Z[i, 0] - Z[i, 2]) + e2 / a * (Z[i, 1] - Z[i, 2])
            depth.scatter_reduce_(0, p, z, "amin")
    return depth.reshape(H, W)


def _project(vp, p, W, H):
    """Clip-space transform of points [..., 4] and the viewport mapping."""
    q = p @ vp.reshape(4, 4)
    w = q[..., 3]
    return torch.stack([(q[..., 0] / w + 1.0) * (0.5 * W), (q[..., 1] / w + 1.0) * (0.5 * H), q[..., 2] / w], -1)


def _exact_raster(case, seed, sc=None):
    dev = _dev()
    sc = _raster_scene(case, seed) if sc is None else sc
    if isinstance(sc, dict) and "xyz" in sc:
        W, H = sc["W"], sc["H"]
        screen = torch.from_numpy(sc["xyz"]).to(dev).double().reshape(-1, 3, 3)
    else:
        if isinstance(sc, dict):
            W, H, vp = sc["W"], sc["H"], sc["view_proj"]
            p = torch.from_numpy(sc["xyz_world"]).to(dev).double().reshape(-1, 3, 3)
        else:
            W, H, vp = sc.W, sc.H, sc.view_proj
            p = torch.from_numpy(sc.pos).to(dev).double().transpose(0, 1)[..., :3]
        p = torch.cat([p, torch.ones_like(p[..., :1])], -1)
        screen = _project(torch.from_numpy(vp).to(dev).double(), p, W, H)
    return _raster_depth(W, H, screen)


def _bernstein(t):
    return torch.stack([(1 - t) ** 3, 3 * t * (1 - t) ** 2, 3 * t * t * (1 - t), t ** 3], -1)


def _jitter(seed, x, y, k):
    """The sampler's integer hash (24 bits) as a fraction."""
    m = 0xFFFFFFFF
    h = (seed * 0x9E3779B1) & m
    h = h ^ ((x * 0x85EBCA77) & m) ^ ((y * 0xC2B2AE3D) & m) ^ ((k * 0x27D4EB2F) & m)
    h = h ^ (h >> 16)
    h = (h * 0x7FEB352D) & m
    h = h ^ (h >> 15)
    h = (h * 0x846CA68B) & m
    h = h ^ (h >> 16)
    return (h >> 8).double() / (1 << 24)


def _exact_reyes(case, seed):
    """Depth buffer of the Reyes frame: split until both screen extents are
    below the threshold, dice, the mean corner depth of every micropolygon
    whose four edges enclose a sample, the nearest depth of a pixel's samples."""
    dev = _dev()
    sc = _reyes_scene(case, seed)
    W, H, spp = sc.W, sc.H, case["spp"]
    thr = case["thr"] if case["thr"] > 0 else 4.0
    levels = case["splits"] if case["splits"] > 0 else 20
    vp = torch.from_numpy(sc.view_proj).to(dev).double()
    P = torch.from_numpy(sc.patches).to(dev).double().reshape(-1, 4, 4, 4)   # [patch, v, u, xyzw]
    half = torch.tensor([[8, 0, 0, 0], [4, 4, 0, 0], [2, 4, 2, 0], [1, 3, 3, 1]], dtype=torch.float64, device=dev) / 8
    other = half.flip(0).flip(1)
    leaves = []
    for level in range(levels + 1):
        s = _project(vp, P, W, H)[..., :2]
        ue = (s[:, :, 1:] - s[:, :, :-1]).norm(dim=-1).sum(2).amax(1)
        ve = (s[:, 1:] - s[:, :-1]).norm(dim=-1).sum(1).amax(1)
        split = ((ue >= thr) | (ve >= thr)) & (level < levels)
        leaves.append((P[~split], ue[~split], ve[~split]))
        along_u, P = (ue >= thr)[split], P[split]
        if P.shape[0] == 0:
            break
        U, V = P[along_u], P[~along_u]
        P = torch.cat([torch.einsum("ij,pvjc->pvic", m, U) for m in (half, other)] +
                      [torch.einsum("ij,pjuc->piuc", m, V) for m in (half, other)])
    P, ue, ve = (torch.cat(v) for v in zip(*leaves))
    if case["grid"] > 0:
        nu = nv = torch.full((P.shape[0],), case["grid"], dtype=torch.int64, device=dev)
    else:
        nu, nv = ((2.0 ** torch.ceil(torch.log2(torch.ceil(e / thr) + 1))).to(torch.int64).clamp(2, 32) for e in (ue, ve))
    depth = torch.ones(W * H, dtype=torch.float64, device=dev)
    xe, ye = W // 64 * 64, H // 64 * 64     # whole 64x64 bins only
    for a, b in torch.unique(torch.stack([nu, nv], 1), dim=0).tolist():
        Q = P[(nu == a) & (nv == b)]
        bu = _bernstein(torch.arange(a + 2, device=dev).double() / a)
        bv = _bernstein(torch.arange(b + 2, device=dev).double() / b)
        for q in Q.split(4096):
            g = _project(vp, torch.einsum("kj,li,pijc->pklc", bu, bv, q), W, H)   # [patch, u, v, xyz]
            c = torch.stack([g[:, :-1, :-1], g[:, 1:, :-1], g[:, 1:, 1:], g[:, :-1, 1:]], 3).reshape(-1, 4, 3)
            z = c[..., 2].mean(1)
            x0, x1 = c[..., 0].amin(1).floor().clamp(0, xe), c[..., 0].amax(1).ceil().clamp(0, xe)
            y0, y1 = c[..., 1].amin(1).floor().clamp(0, ye), c[..., 1].amax(1).ceil().clamp(0, ye)
            some = (x1 > x0) & (y1 > y0) & (z <= 1.0)
            c, z, x0, x1, y0, y1 = (v[some] for v in (c, z, x0, x1, y0, y1))
            if not z.numel():
                continue
            x0, y0 = x0.to(torch.int64), y0.to(torch.int64)
            d = c.roll(-1, 1) - c
            for i, x, y in _expand(x1.to(torch.int64) - x0, y1.to(torch.int64) - y0):
                x, y = x + x0[i], y + y0[i]
                for k in range(spp):
                    if spp == 1:
                        px, py = x + 0.5, y + 0.5
                    else:
                        px = x + ((k & 1) + _jitter(7, x, y, 2 * k)) * 0.5
                        py = y + ((k >> 1) + _jitter(7, x, y, 2 * k + 1)) * 0.5
                    e = [(py - c[i, j, 1]) * d[i, j, 0] - (px - c[i, j, 0]) * d[i, j, 1] for j in range(4)]
                    cov = ((e[0] > 0) & (e[1] > 0) & (e[2] > 0) & (e[3] > 0)) | \
                          ((e[0] < 0) & (e[1] < 0) & (e[2] < 0) & (e[3] < 0))
                    depth.scatter_reduce_(0, (y * W + x)[cov], z[i[cov]], "amin")
    return depth.reshape(H, W)


def exact(case, seed):
    if case["kind"] == "mix":
        return [(None, _exact_raster(case, seed, pk.scenes.plain_scene(n=n, W=W, H=H, seed=1000 * (seed + 1) + i)))
                for i, (n, W, H) in enumerate(_mix_sizes(case))]
    if case["kind"] == "reyes":
        return [(None, _exact_reyes(case, seed))]
    d = _exact_raster(case, seed)
    if case["form"] == "app":
        return None, d.reshape(-1)
    return (None, d) if case["form"] == "upload" else [(None, d)]
