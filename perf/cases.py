"""The work that users of fallingsand3d_gb300 have it do, as measurable cases.

Every case is one pass through the package's public entry points.  The kinds,
and what each stands for in real use:

* grid     the drop-in step on a caller's own uint8 grid in device memory;
* job      a drop-in run: a level's grid in device memory taken through n
           steps by one call, in place (with the static scratch, `noalloc`,
           for callers whose allocator owns the GPU);
* session  a whole run from host memory: world from a numpy grid, n steps,
           read back (one simulation asked for by a script);
* live     a long-lived pool of mixed worlds: one more segment of every world
           and a snapshot of all of them into device memory (the worlds go on
           from pass to pass);
* rollout  a pool used for data generation: fresh worlds from device grids
           admitted together, a few segments, final grids back to device memory;
* hosted   the same for grids in page-locked host memory, through the
           asynchronous admission and read-back;
* serve    a burst of simulation requests through the serving loop;
* play     an engine's frame loop: a library-owned world stepped once and
           drawn (voxel traversal) per pass, frame after frame (the world goes
           on from pass to pass, as it does in a game);
* scene    the upstream scene's frame: its cube-grid meshes, its raymarched
           object and its full-screen sphere shader.

Sizes are those of the package's workloads (64^3 parity worlds, 512^3 pillars,
mixed worlds with sides of 16 to 128, 1024^3 dunes, 1920x1080 frames) and
generic odd ones around them.  In the kinds with a level to start from, each
pass starts again from that level.
"""
import math

import numpy as np
import torch

import fallingsand3d_gb300 as fs

SIDES = (16, 24, 32, 48, 64, 96, 128)  # sides of the mixed pool worlds

# the scene's cube: corners and faces of +-1 (the faces' diagonals matter to the object's material)
_CORNERS = np.array([(1, 1, -1), (1, -1, -1), (1, 1, 1), (1, -1, 1), (-1, 1, -1), (-1, -1, -1), (-1, 1, 1), (-1, -1, 1)])
_FACES = np.array([(5, 3, 1), (3, 8, 4), (7, 6, 8), (2, 8, 6), (1, 4, 2), (5, 2, 6),
                   (5, 7, 3), (3, 7, 8), (7, 5, 6), (2, 4, 8), (1, 3, 4), (5, 1, 2)])
CUBE = _CORNERS[_FACES - 1].astype(np.float32)  # 12 x 3 x 3


def listed():
    return [
        # the smallest pass there is: one frame of a small world in a small window
        {"name": "play_64", "kind": "play", "X": 64, "Y": 64, "Z": 64, "W": 320, "H": 180},
        # an engine's own grid of odd size, a few steps per call
        {"name": "grid_ragged", "kind": "grid", "X": 75, "Y": 61, "Z": 93, "steps": 8, "statics": True},
        # the single large drop-in world: 512^3, stone pillars under falling sand and water
        {"name": "grid_512", "kind": "grid", "X": 512, "Y": 512, "Z": 512, "steps": 32, "statics": False},
        # a small drop-in run of a few seconds of game time
        {"name": "job_96", "kind": "job", "X": 96, "Y": 80, "Z": 112, "steps": 200, "statics": False, "noalloc": False},
        # a mid-size drop-in run with walls of a custom material, no allocation allowed
        {"name": "job_400", "kind": "job", "X": 400, "Y": 300, "Z": 350, "steps": 100, "statics": True, "noalloc": True},
        # a script's run of one world from and to host memory
        {"name": "session_128", "kind": "session", "X": 128, "Y": 96, "Z": 110, "steps": 100, "statics": False},
        # the pool in its steady state: 2048 mixed worlds
        {"name": "live_2048", "kind": "live", "worlds": 2048, "mix": 1, "ragged": False, "age": 640},
        # data generation: 512 fresh mixed worlds, 128 steps each
        {"name": "rollout_512", "kind": "rollout", "worlds": 512, "mix": 2, "ragged": False, "segments": 2},
        # worlds of odd sizes that come from and go back to the host
        {"name": "hosted_256", "kind": "hosted", "worlds": 256, "mix": 3, "ragged": True, "segments": 1},
        # a burst of requests, 10 to 1000 steps each
        {"name": "serve_1000", "kind": "serve", "requests": 1000},
        # the largest world, stepped and drawn frame after frame
        {"name": "play_1024", "kind": "play", "X": 1024, "Y": 1024, "Z": 1024, "W": 1920, "H": 1080},
        # the upstream scene at full HD: 5202 cubes, the object, the shader
        {"name": "scene_1080", "kind": "scene", "cubes": 51, "W": 1920, "H": 1080},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, sizes spread over their ranges."""
    kind = rng.choice(("grid", "job", "session", "live", "rollout", "hosted", "serve", "play", "scene"))
    side = lambda lo, hi: {a: _log_int(rng, lo, hi) for a in ("X", "Y", "Z")}  # noqa: E731
    if kind == "grid":
        d = side(24, 512)
        if rng.random() < 0.5:  # rows of whole words, as engines often have
            d["X"] = max(16, d["X"] // 16 * 16)
        return {"kind": kind, **d, "steps": _log_int(rng, 1, 32), "statics": rng.random() < 0.5}
    if kind == "job":
        return {"kind": kind, **side(24, 400), "steps": _log_int(rng, 4, 200), "statics": rng.random() < 0.5,
                "noalloc": rng.random() < 0.3}
    if kind == "session":
        return {"kind": kind, **side(24, 160), "steps": _log_int(rng, 4, 200), "statics": rng.random() < 0.5}
    if kind == "live":
        return {"kind": kind, "worlds": _log_int(rng, 16, 1500), "mix": rng.randrange(1, 1 << 20),
                "ragged": rng.random() < 0.5, "age": rng.choice((0, 128, 640))}
    if kind == "rollout":
        return {"kind": kind, "worlds": _log_int(rng, 8, 512), "mix": rng.randrange(1, 1 << 20),
                "ragged": rng.random() < 0.5, "segments": rng.choice((1, 2, 3))}
    if kind == "hosted":
        return {"kind": kind, "worlds": _log_int(rng, 8, 256), "mix": rng.randrange(1, 1 << 20),
                "ragged": rng.random() < 0.5, "segments": rng.choice((1, 2))}
    if kind == "serve":
        return {"kind": kind, "requests": _log_int(rng, 50, 1000)}
    if kind == "play":
        W = _log_int(rng, 320, 1920)
        return {"kind": kind, **side(48, 640), "W": W, "H": W * 9 // 16}
    W = _log_int(rng, 320, 1920)
    return {"kind": kind, "cubes": _log_int(rng, 3, 51), "W": W, "H": W * 9 // 16}


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _fill(g, gen, sand, water, from_y):
    """Sand and water, cell by cell, into the layers from from_y up."""
    step = max(1, (1 << 26) // max(1, g.shape[1] * g.shape[2]))
    for y in range(from_y, g.shape[0], step):
        part = g[y:y + step]
        u = torch.rand(part.shape, generator=gen, device="cuda")
        new = torch.where(u < sand, 2, torch.where(u < sand + water, 3, 0)).to(torch.uint8)
        part.copy_(torch.where(part == 0, new, part))


def _level(X, Y, Z, seed, statics):
    """A level: a stone floor, stone pillars, the upper 60 % filled with loose
    sand and water; with `statics`, thin walls of a custom material."""
    gen = _generator(seed)
    g = torch.zeros((Y, Z, X), dtype=torch.uint8, device="cuda")
    g[:2] = 1
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    for _ in range(max(1, X * Z // 1024)):
        w, h = r.randint(2, 9), r.randint(max(1, Y // 50), max(2, 6 * Y // 10))
        x, z = r.randint(0, X), r.randint(0, Z)
        g[2:2 + h, z:z + w, x:x + w] = 1
    if statics:
        for _ in range(4):
            y, z = r.randint(2, max(3, Y // 2)), r.randint(0, Z)
            g[2:y, z:z + 1, :] = 5
            g[2:y, :, r.randint(0, X)] = 4
    _fill(g, gen, 0.30, 0.10, 2 * Y // 5)
    return g


def _dunes(X, Y, Z, seed):
    """Sand dunes (smooth heights up to 30 % of Y) under rain (10 % water)."""
    gen = _generator(seed)
    h = torch.zeros((1, 1, Z, X), device="cuda")
    for octave in range(4):
        n = 4 << octave
        c = torch.rand((1, 1, n + 3, n + 3), generator=gen, device="cuda")
        h += torch.nn.functional.interpolate(c, size=(Z, X), mode="bicubic", align_corners=True) / (1 << octave)
    top = (h[0, 0] / 1.875 * 0.3 * Y).round().clamp(0, Y).to(torch.int32)
    g = torch.empty((Y, Z, X), dtype=torch.uint8, device="cuda")
    y = torch.arange(Y, device="cuda", dtype=torch.int32).view(-1, 1, 1)
    step = max(1, (1 << 26) // (X * Z))
    for a in range(0, Y, step):
        rain = torch.rand(g[a:a + step].shape, generator=gen, device="cuda") < 0.1
        g[a:a + step] = torch.where(y[a:a + step] < top, 2, torch.where(rain, 3, 0)).to(torch.uint8)
    return g


def _pool_dims(case):
    """Sides of the pool's worlds: of the usual choice, or any from 10 to 130."""
    r = np.random.RandomState(case["mix"])
    n = case["worlds"]
    if case["ragged"]:
        return np.exp(r.uniform(math.log(10), math.log(130), (n, 3))).astype(np.int64)  # X, Y, Z
    return r.choice(SIDES, (n, 3)).astype(np.int64)


def _arena(dims):
    """Offsets of the worlds' grids in one buffer, each at a multiple of 16 bytes, and its size."""
    cells = dims.prod(axis=1)
    ends = np.cumsum((cells + 15) // 16 * 16)
    return np.concatenate([[0], ends[:-1]]), int(ends[-1])


def _pool_grids(dims, offs, size, seed):
    """The fresh worlds of a pool on the device: a floor and a random filling above the middle."""
    gen, r = _generator(seed), np.random.RandomState(seed & 0x7FFFFFFF)
    buf = torch.zeros(size, dtype=torch.uint8, device="cuda")
    for (X, Y, Z), o in zip(dims.tolist(), offs.tolist()):
        g = buf[o:o + X * Y * Z].view(Y, Z, X)
        g[:2] = 1
        _fill(g, gen, r.uniform(0.05, 0.4), r.uniform(0.0, 0.2), Y // 2)
    return buf


class _DeviceArray:
    """Device memory of a world as an array (for torch.as_tensor); it keeps the
    world, and so the memory, for as long as the tensor lives."""

    def __init__(self, world, shape, typestr):
        self.world = world
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (world.device_ptr(), False), "version": 3}


def _planes(world):
    n = world.Y * world.Z * ((world.X + 63) // 64) * 4
    t = torch.as_tensor(_DeviceArray(world, (n,), "<i4"), device="cuda")
    t.world = world  # the tensor itself keeps it too
    return t


def _scene_view(case, seed):
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    return {"cam_pos": (float(r.uniform(-2, 2)), float(r.uniform(-5, -3)), float(-case["cubes"] / 2 - r.uniform(6, 8))),
            "rot_y": float(r.uniform(-8, 8))}, {"rot_y": float(r.uniform(-30, 30))}, r.uniform(-0.3, 0.3, 2)


def _cube_vertices():
    f = CUBE.reshape(-1, 3)
    return np.c_[f, (f[:, [0, 2]] + 1) * 0.5].astype(np.float32)


def _cube_places(n):
    return [(x - n // 2, y, z - n // 2) for y in (0, 5) for x in range(n) for z in range(n)]


def _texture(seed):
    return np.random.RandomState((seed + 1) & 0x7FFFFFFF).randint(0, 256, (512, 512, 4)).astype(np.uint8)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case, "seed": seed}
    if kind in ("grid", "job"):
        s["level"] = _level(case["X"], case["Y"], case["Z"], seed, case["statics"])
        s["grid"] = torch.empty_like(s["level"])
        s["stream"] = torch.cuda.current_stream().cuda_stream
    elif kind == "session":
        s["level"] = _level(case["X"], case["Y"], case["Z"], seed, case["statics"]).cpu().numpy()
    elif kind == "live":
        dims = _pool_dims(case)
        offs, size = _arena(dims)
        first = _pool_grids(dims, offs, size, seed)
        torch.cuda.synchronize()
        b = fs.Batch(64 << 30)
        s["batch"], s["out"] = b, first  # the snapshots take the place of the first grids
        seeds = np.arange(len(dims), dtype=np.uint64) + np.uint64(seed)
        s["ptrs"] = offs.astype(np.uint64) + np.uint64(first.data_ptr())
        s["tickets"] = b.admit_many(None, seeds, 1 << 40, ptrs=s["ptrs"], dims=dims)
        for _ in range(case["age"] // 64):
            b.run_segment()
        b.sync()
    elif kind in ("rollout", "hosted"):
        dims = _pool_dims(case)
        offs, size = _arena(dims)
        grids = _pool_grids(dims, offs, size, seed)
        if kind == "hosted":
            host = torch.empty(size, dtype=torch.uint8, pin_memory=True)
            host.copy_(grids)
            grids, out = host, torch.zeros(size, dtype=torch.uint8, pin_memory=True)
        else:
            out = torch.zeros_like(grids)
        s.update(grids=grids, out=out, dims=dims, batch=fs.Batch(64 << 30),
                 seeds=np.arange(len(dims), dtype=np.uint64) + np.uint64(seed),
                 src=offs.astype(np.uint64) + np.uint64(grids.data_ptr()),
                 dst=offs.astype(np.uint64) + np.uint64(out.data_ptr()))
        torch.cuda.synchronize()
    elif kind == "serve":
        # every request arrives at once: the loop runs at its capacity
        s["params"] = fs.serve_params(1e9, 1.0, master_seed=seed, max_requests=case["requests"])
    elif kind == "play":
        g = _dunes(case["X"], case["Y"], case["Z"], seed).cpu().numpy()
        s["world"] = fs.World(g, seed)
        s["planes"] = _planes(s["world"])
        s["cam"] = fs.camera_world_view(case["X"], case["Y"], case["Z"], case["W"], case["H"])
        s["image"] = torch.zeros((case["H"], case["W"], 4), device="cuda")
        s["world"].step(16)  # some way into the run, the traversal's map built
        s["world"].render(s["cam"], case["W"], case["H"], out_ptr=s["image"].data_ptr())
        s["world"].sync()
    elif kind == "scene":
        mesh_kw, object_kw, sphere = _scene_view(case, seed)
        s["vertices"] = torch.from_numpy(_cube_vertices()).cuda()
        s["texture"] = torch.from_numpy(_texture(seed)).cuda()
        draws = []
        for x, y, z in _cube_places(case["cubes"]):
            m = np.diag([0.2, 0.2, 0.2, 1.0])
            m[:3, 3] = (x, y, z)
            mat, col = (fs.MAT_TEXTURED, (1.0, 0.0, 0.0, 1.0)) if y else (fs.MAT_BASIC, (0.0, 1.0, 0.0, 1.0))
            draws.append(fs.mesh_draw(s["vertices"].data_ptr(), 36, mat, m, col, s["texture"].data_ptr() if y else 0, 512, 512))
        s["draws"] = fs.mesh_draws(draws)
        s["mesh_view"], s["object_view"] = fs.object_view_scene(**mesh_kw), fs.object_view_scene(**object_kw)
        s["cube"], s["cam"] = CUBE, fs.camera_fs_raymarch()
        s["cam"].origin[0], s["cam"].origin[1] = float(sphere[0]), float(sphere[1])
        s["stream"] = torch.cuda.current_stream().cuda_stream
        s["images"] = {k: torch.zeros((case["H"], case["W"], 4), device="cuda") for k in ("mesh", "object", "sphere")}
    else:
        raise ValueError(kind)
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "grid":
        s["grid"].copy_(s["level"])
        fs.step_device(s["grid"].data_ptr(), c["X"], c["Y"], c["Z"], s["seed"], 0, c["steps"], s["stream"])
        return s["grid"]
    if kind == "job":
        s["grid"].copy_(s["level"])
        a = (s["grid"].data_ptr(), c["X"], c["Y"], c["Z"], s["seed"], 0, c["steps"], s["stream"])
        if c["noalloc"]:
            fs.check(fs.lib().fs3d_run_device_noalloc(*a))
        else:
            fs.run_device(*a)
        return s["grid"]
    if kind == "session":
        with fs.World(s["level"], s["seed"]) as w:
            w.step(c["steps"])
            return w.read()
    if kind == "live":
        s["batch"].run_segment()
        s["batch"].read_many(s["tickets"], s["ptrs"])
        return s["out"]
    if kind == "rollout":
        t = s["batch"].admit_many(None, s["seeds"], 64 * c["segments"], ptrs=s["src"], dims=s["dims"])
        for _ in range(c["segments"]):
            s["batch"].run_segment()
        s["batch"].retire_many(t, s["dst"])
        return s["out"]
    if kind == "hosted":
        t = s["batch"].admit_many(None, s["seeds"], 64 * c["segments"], ptrs=s["src"], dims=s["dims"], wait=False)
        for _ in range(c["segments"]):
            s["batch"].run_segment()
        s["batch"].retire_many(t, s["dst"], wait=False)
        s["batch"].wait_copies()
        return s["out"]
    if kind == "serve":
        _, reqs = fs.serve(s["params"])
        return np.array([[q.X, q.Y, q.Z, q.n_steps] for q in reqs]), np.array([q.hash for q in reqs], np.uint64).view(np.int64)
    if kind == "play":
        s["world"].step(1)
        s["world"].render(s["cam"], c["W"], c["H"], out_ptr=s["image"].data_ptr())
        return {"planes": s["planes"], "image": s["image"]}
    im = s["images"]
    fs.render_meshes_device(s["mesh_view"], s["draws"], c["W"], c["H"], im["mesh"].data_ptr(), s["stream"])
    fs.render_object_device(s["object_view"], s["cube"], c["W"], c["H"], im["object"].data_ptr(), s["stream"])
    fs.render_sdf_device(s["cam"], c["W"], c["H"], im["sphere"].data_ptr(), s["stream"])
    return im


def work(case):
    """Bytes: the grids (1 byte a cell) or the world's state (2 bits a cell)
    read once and written once, frames written once.  No floating-point
    operations but the frames' (a handful per pixel), which are left out."""
    kind = case["kind"]
    if "X" in case:
        cells = case["X"] * case["Y"] * case["Z"]
    if kind in ("grid", "job", "session"):
        return {"bytes": 2 * cells, "flops": 0}
    if kind == "live":
        return {"bytes": int(_pool_dims(case).prod(axis=1).sum() * 3 // 2), "flops": 0}
    if kind in ("rollout", "hosted"):
        return {"bytes": int(_pool_dims(case).prod(axis=1).sum() * 2), "flops": 0}
    if kind == "serve":  # worlds of 301 000 cells in the mean, made, run and hashed in 2 bits a cell
        return {"bytes": case["requests"] * 301000 // 2, "flops": 0}
    if kind == "play":
        return {"bytes": cells // 2 + 16 * case["W"] * case["H"], "flops": 0}
    return {"bytes": 3 * 16 * case["W"] * case["H"] + 2 * case["cubes"] ** 2 * 128, "flops": 0}


# ---------------------------------------------------------------- frames in 64 bits
def _rot_translate(cam_pos, rot_y):
    a = math.radians(rot_y)
    R = np.array([[math.cos(a), 0, math.sin(a), 0], [0, 1, 0, 0], [-math.sin(a), 0, math.cos(a), 0], [0, 0, 0, 1.0]])
    T = np.eye(4)
    T[:3, 3] = cam_pos
    return R @ T


def _projection():
    """70 degrees, aspect 1700/900, depth 0.01 to 200 (OpenGL's range), y negated."""
    th, n, f = math.tan(math.radians(35.0)), 0.01, 200.0
    P = np.zeros((4, 4))
    P[0, 0], P[1, 1] = 1 / (1700 / 900 * th), -1 / th
    P[2, 2], P[2, 3], P[3, 2] = -(f + n) / (f - n), -2 * f * n / (f - n), -1.0
    return P


def _raster(tri, mvp_of, W, H, dev):
    """Nearest triangle per pixel centre: (triangle index or -1, barycentric
    weights, the triangles' clip w).  tri: T x 3 x 4 clip coordinates."""
    clip = torch.einsum("tij,tkj->tki", mvp_of, tri)
    w = clip[..., 3]
    sx, sy = clip[..., 0] / w * (W / 2) + W / 2, clip[..., 1] / w * (H / 2) + H / 2
    sz = clip[..., 2] / w
    x0, x1 = sx.amin(1).floor().clamp(0, W).long(), sx.amax(1).ceil().clamp(-1, W - 1).long()
    y0, y1 = sy.amin(1).floor().clamp(0, H).long(), sy.amax(1).ceil().clamp(-1, H - 1).long()
    nx, ny = (x1 - x0 + 1).clamp(min=0), (y1 - y0 + 1).clamp(min=0)
    count = nx * ny
    depth = torch.full((W * H,), math.inf, dtype=torch.float64, device=dev)
    owner = torch.full((W * H,), -1, dtype=torch.int64, device=dev)
    weights = torch.zeros((W * H, 3), dtype=torch.float64, device=dev)
    ends = count.cumsum(0)
    first = 0
    while first < len(count):
        base = int(ends[first - 1]) if first else 0
        last = max(first + 1, int(torch.searchsorted(ends, torch.tensor(base + 4_000_000, device=dev))))
        t = torch.repeat_interleave(torch.arange(first, last, device=dev), count[first:last])
        i = torch.arange(len(t), device=dev) - (ends[t] - count[t] - base)
        px, py = x0[t] + i % nx[t].clamp(min=1), y0[t] + i // nx[t].clamp(min=1)
        fx, fy = px + 0.5, py + 0.5
        e = []
        for a, b in ((1, 2), (2, 0), (0, 1)):
            e.append((sx[t, b] - sx[t, a]) * (fy - sy[t, a]) - (sy[t, b] - sy[t, a]) * (fx - sx[t, a]))
        e = torch.stack(e, 1)
        area = e.sum(1)
        l = e / area[:, None]
        z = (l * sz[t]).sum(1)
        ok = (l >= 0).all(1) & (area != 0) & (z >= 0) & (z <= 1)
        t, l, z, p = t[ok], l[ok], z[ok], (py * W + px)[ok]
        best = depth.clone().scatter_reduce_(0, p, z, "amin")
        win = z == best[p]
        owner[p[win]], weights[p[win]], depth = t[win], l[win], best
        first = last
    return owner, weights, w


def _mesh_image(case, seed, dev):
    W, H = case["W"], case["H"]
    mesh_kw, _, _ = _scene_view(case, seed)
    v = torch.tensor(_cube_vertices(), dtype=torch.float64, device=dev)
    places = torch.tensor(_cube_places(case["cubes"]), dtype=torch.float64, device=dev)
    n = len(places)
    pos = (v[None, :, :3] * 0.2 + places[:, None]).reshape(-1, 3, 3)
    tri = torch.cat([pos, torch.ones_like(pos[..., :1])], 2)
    vp = torch.tensor(_projection() @ _rot_translate(**mesh_kw), device=dev)
    owner, l, w = _raster(tri, vp.expand(len(tri), 4, 4), W, H, dev)
    img = torch.tensor([0.0, 0, 1, 1], dtype=torch.float64, device=dev).repeat(W * H, 1)
    hit = owner >= 0
    o, l = owner[hit], l[hit] / w[owner[hit]]
    uv = torch.einsum("pk,pkc->pc", l, v[:, 3:].repeat(n, 1).reshape(-1, 3, 2)[o]) / l.sum(1, keepdim=True)
    c = torch.arange(256, dtype=torch.float64, device=dev) / 255
    lut = torch.where(c <= 0.04045, c / 12.92, ((c + 0.055) / 1.055) ** 2.4)
    ij = (uv * 512).floor().long() % 512
    texel = lut[torch.from_numpy(_texture(seed)).to(dev)[ij[:, 1], ij[:, 0]][:, :3].long()]
    red = torch.cat([texel + torch.tensor([1.0, 0, 0], device=dev), torch.ones_like(texel[:, :1])], 1).clamp(0, 1)
    green = torch.tensor([0.0, 1, 0, 1], dtype=torch.float64, device=dev)
    img[hit] = torch.where((o // 12 >= n // 2)[:, None], red, green)
    return img.view(H, W, 4)


def _march(o, d, sdf):
    """Sphere tracing as the shaders do it: (hit, distance along the ray, steps taken)."""
    t = torch.zeros_like(d[..., 0])
    hit, gone, steps = torch.zeros_like(t, dtype=torch.bool), torch.zeros_like(t, dtype=torch.bool), torch.zeros_like(t)
    for _ in range(64):
        dist = sdf(o + d * t[..., None])
        on = ~hit & ~gone
        hit |= on & (dist < 0.001)
        gone |= on & ~hit & (t > 1000)
        on &= ~hit & ~gone
        t, steps = torch.where(on, t + dist, t), torch.where(on, steps + 1, steps)
    return hit, t, steps


def _object_image(case, seed, dev):
    W, H = case["W"], case["H"]
    _, kw, _ = _scene_view(case, seed)
    tri3 = torch.tensor(CUBE, dtype=torch.float64, device=dev)
    tri = torch.cat([tri3, torch.ones_like(tri3[..., :1])], 2)
    mvp = torch.tensor(_projection() @ _rot_translate((0, 0, -5.0), kw["rot_y"]), device=dev)
    owner, l, _ = _raster(tri, mvp.expand(len(tri), 4, 4), W, H, dev)
    img = torch.tensor([0.0, 0, 1, 1], dtype=torch.float64, device=dev).repeat(W * H, 1)
    hit = owner >= 0
    o = torch.tensor([0.0, 0, 5], dtype=torch.float64, device=dev)
    d = torch.einsum("pk,pkc->pc", l[hit], tri3[owner[hit]]) - o
    d = d / d.norm(dim=1, keepdim=True)

    def box(p):
        q = p.abs() - 0.5
        return q.clamp(min=0).norm(dim=-1) + q.amax(-1).clamp(max=0)

    on, _, steps = _march(o, d, box)
    col = torch.zeros((len(d), 4), dtype=torch.float64, device=dev)
    col[:, 3] = 1
    col[:, 0] = torch.where(on, (1 - 0.05 * steps).clamp(min=0.05), torch.zeros_like(steps))
    img[hit] = col
    return img.view(H, W, 4)


def _sphere_image(case, seed, dev):
    W, H = case["W"], case["H"]
    _, _, at = _scene_view(case, seed)
    f = dict(dtype=torch.float64, device=dev)
    x = (1 - (torch.arange(W, **f) + 0.5) / W) * 2 - 1
    y = ((torch.arange(H, **f) + 0.5) / H * 2 - 1) / (1700 / 900)
    d = torch.stack([x.expand(H, W), y[:, None].expand(H, W), torch.ones((H, W), **f)], 2)
    d = d / d.norm(dim=2, keepdim=True)
    o, light = torch.tensor([at[0], at[1], -5.0], **f), torch.tensor([2.0, 5.0, 3.0], **f)
    hit, t, _ = _march(o, d, lambda p: p.norm(dim=-1) - 0.5)
    p = o + d * t[..., None]
    n = p / p.norm(dim=2, keepdim=True)
    ld = p - light
    diff = (n * ld / ld.norm(dim=2, keepdim=True)).sum(2).clamp(min=0.05)
    img = torch.zeros((H, W, 4), **f)
    img[..., 0], img[..., 3] = torch.where(hit, diff, torch.zeros_like(diff)), 1
    return img


def exact(case, seed):
    """The scene's frames in 64 bits.  The other kinds give whole numbers (and
    a frame of a world that only those determine)."""
    if case["kind"] != "scene":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return {"mesh": _mesh_image(case, seed, dev), "object": _object_image(case, seed, dev),
            "sphere": _sphere_image(case, seed, dev)}
