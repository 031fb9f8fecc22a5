"""Timed cases: what a program that uses this library has it do.

A case is a dict of plain values; ``prepare`` makes what such a program holds
before the call (sessions with a map under way, the frames that come next) and
``run`` makes one pass through the public entry points and returns what they
give.  The kinds:

* ``frame``  one camera, one frame: System.process_images (or the staged form
             from pinned host memory), the camera pose and the shaded preview
* ``tick``   a server's tick: FusionBatch.process over all sessions, the next
             frames staged from pinned host memory meanwhile, the tick's
             results, and the preview of one session
* ``fuse``   mapping with poses from elsewhere: DenseMapping.update, then the
             raycast with the model normals
* ``track``  odometry alone: both image pyramids and compute_transform
* ``view``   a free viewpoint into a large map: raycast_check_visibility, the
             raycast with normals and colours, and the shading
* ``mesh``   the mesh of a whole map, with normals or colours
* ``park``   a paused session evicted to pinned host memory and resumed in
             another arena, pruned around the camera, and its next frame fused

The frames are the library's synthetic rooms (a 1.5 m circle through a 4 x 4 x 3 m
room, or the figure-eight of the 8 x 8 x 3 m one), played forwards and backwards
so that the camera moves continuously however many passes are made.
"""
import math

import numpy as np
import torch

import libfusion_gb300 as L

LAYOUTS = {"ref": L.VOXEL_REF, "half": L.VOXEL_HALF, "snorm": L.VOXEL_SNORM}


def listed():
    return [
        # a small robot's or phone's camera at 320x240, the default voxel size and layout: launches and latency
        dict(name="frame_qvga", kind="frame", width=320, height=240, voxel=0.01, layout="ref", levels=3, host=False),
        # the ordinary depth camera, fine voxels, frames arriving in pinned host memory
        dict(name="frame_vga", kind="frame", width=640, height=480, voxel=0.005, layout="snorm", levels=3, host=True),
        # a 1280x720 camera with a four-level pyramid
        dict(name="frame_hd", kind="frame", width=1280, height=720, voxel=0.008, layout="half", levels=4, host=False),
        # a server with a few cameras: the tick of the low-load hours
        dict(name="tick_few", kind="tick", width=640, height=480, sessions=4, layout="snorm"),
        # a full server: 64 cameras of 640x480 with 5, 6, 8 and 10 mm voxels
        dict(name="tick_many", kind="tick", width=640, height=480, sessions=64, layout="snorm"),
        # offline reconstruction from known poses
        dict(name="fuse_vga", kind="fuse", width=640, height=480, voxel=0.005, layout="ref", normals=False),
        # the normal-weighted update of a camera whose size is no multiple of the kernels' tiles
        dict(name="fuse_ragged", kind="fuse", width=328, height=248, voxel=0.01, layout="snorm", normals=True),
        # odometry without a map: a small and a large camera
        dict(name="track_qvga", kind="track", width=320, height=240, levels=3),
        dict(name="track_hd", kind="track", width=1280, height=720, levels=3),
        # an operator looking around in a large map
        dict(name="view_vga", kind="view", width=640, height=480, voxel=0.005, layout="snorm", frames=40),
        # a finished map meshed for download, with normals
        dict(name="mesh_large", kind="mesh", blocks=48000, voxel=0.005, layout="snorm", mode="normal"),
        # a camera pauses: parked, resumed, trimmed, and on with the next frame
        dict(name="park_vga", kind="park", width=640, height=480, voxel=0.008, layout="snorm"),
    ]


def _spread(rng, lo, hi):
    """A number between lo and hi, spread over the logarithm."""
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi, step=8):
    w = int(_spread(rng, lo, hi)) // step * step
    h = int(w * rng.choice([0.5625, 0.625, 0.75])) // step * step
    return w, max(h, 96)


def draw(rng):
    kind = rng.choice(["frame", "frame", "tick", "fuse", "track", "view", "mesh", "park"])
    layout = rng.choice(sorted(LAYOUTS))
    if kind == "mesh":
        return dict(kind=kind, blocks=int(_spread(rng, 300, 40000)), voxel=rng.choice([0.005, 0.008, 0.01]),
                    layout=layout, mode=rng.choice(["vertex", "normal", "colour"]))
    if kind == "tick":
        w, h = _size(rng, 256, 900)
        return dict(kind=kind, width=w, height=h, sessions=int(_spread(rng, 2, 33)), layout=layout)
    levels = rng.choice([2, 3, 4]) if kind in ("frame", "track") else 3
    w, h = _size(rng, 192, 1288, 2 ** max(3, levels))
    if kind == "track":
        return dict(kind=kind, width=w, height=h, levels=levels)
    voxel = rng.choice([0.005, 0.006, 0.008, 0.01, 0.016])
    if kind == "frame":
        return dict(kind=kind, width=w, height=h, voxel=voxel, layout=layout, levels=levels, host=rng.random() < 0.5)
    if kind == "fuse":
        return dict(kind=kind, width=w, height=h, voxel=voxel, layout=layout, normals=rng.random() < 0.5)
    if kind == "view":
        return dict(kind=kind, width=w, height=h, voxel=voxel, layout=layout, frames=rng.randrange(8, 40))
    return dict(kind=kind, width=w, height=h, voxel=voxel, layout=layout)


# ------------------------------------------------------------------ inputs

def _intrinsics(w, h):
    f = 525.0 * w / 640.0
    return L.IntrinsicMatrix(w, h, f, f, (w - 1) / 2.0, (h - 1) / 2.0)


def _config(voxel, layout, levels=3, blocks=1 << 17, **over):
    """The served configuration: a truncation of three voxels within 2 to 5 cm, depths to 4 m."""
    kw = dict(voxel_size=voxel, truncation=min(max(3.0 * voxel, 0.02), 0.05), zmin_update=0.3, zmax_update=4.0,
              zmin_raycast=0.3, zmax_raycast=4.0, num_buckets=4 * blocks, num_blocks=blocks,
              voxel_layout=LAYOUTS[layout], num_levels=levels, max_iterations=[10, 5, 3, 3, 3], max_probe=256)
    kw.update(over)
    return L.default_config(**kw)


def _large_room(seed):
    return L.SynthScene(seed=seed, trajectory=1, room=(8, 8, 3), n_spheres=20, n_boxes=12, radius=2.5, speed=0.5,
                        fps=30)


def _frames(scene, K, ks, pinned=False):
    """Frames `ks` of a scene as (depth u16 mm, rgb8) tensors, on the GPU or in pinned host memory."""
    got = [scene.render(K, k) for k in ks]
    if pinned:
        host = [(torch.empty(d.shape, dtype=d.dtype, pin_memory=True), torch.empty(c.shape, dtype=c.dtype, pin_memory=True))
                for d, c in got]
        for (d, c), (hd, hc) in zip(got, host):
            hd.copy_(d, non_blocking=True)
            hc.copy_(c, non_blocking=True)
        got = host
    torch.cuda.synchronize()
    return got


def _metres(d):
    return d.to(torch.int32).to(torch.float32) * 0.001


class _Player:
    """Indices 0 .. n-1 forwards and backwards without end."""

    def __init__(self, n):
        self.n, self.i = n, 0

    def next(self):
        k = self.i % (2 * self.n - 2)
        self.i += 1
        return k if k < self.n else 2 * self.n - 2 - k


# ------------------------------------------------------------------ prepare

def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def _prepare_frame(case, seed):
    K = _intrinsics(case["width"], case["height"])
    sc = L.SynthScene(seed=seed)
    n = 16
    s = L.System(K, _config(case["voxel"], case["layout"], case["levels"]))
    s.set_pose(sc.pose(0))
    st = dict(kind="frame", s=s, frames=_frames(sc, K, range(n), case["host"]), play=_Player(n), host=case["host"])
    for _ in range(n):  # a map under way
        _run_frame(st)
    return st


def _prepare_tick(case, seed):
    K = _intrinsics(case["width"], case["height"])
    S, n = case["sessions"], 6
    voxels = (0.005, 0.006, 0.008, 0.010)
    sessions, frames = [], []
    b = L.FusionBatch(S)
    for i in range(S):
        sc = L.SynthScene(seed=64 * seed + i)
        s = L.System(K, _config(voxels[i % 4], case["layout"]))
        s.set_pose(sc.pose(0))
        b.set(i, s)
        sessions.append(s)
        frames.append(_frames(sc, K, range(n), pinned=True))
    st = dict(kind="tick", b=b, sessions=sessions, frames=frames, play=_Player(n), copy=torch.cuda.Stream(),
              active=[True] * S, shown=0)
    _stage_tick(st)
    for _ in range(n):
        _run_tick(st)
    return st


def _stage_tick(st):
    k = st["play"].next()
    for i, f in enumerate(st["frames"]):
        st["b"].stage(i, f[k][0], f[k][1], stream=st["copy"])


def _prepare_fuse(case, seed):
    K = _intrinsics(case["width"], case["height"])
    sc = L.SynthScene(seed=seed)
    n = 12
    frames = [(_metres(d), c) for d, c in _frames(sc, K, range(n))]
    m = L.DenseTracking(K, _config(case["voxel"], case["layout"]))
    normals = [None] * n
    if case["normals"]:
        for k, (d, c) in enumerate(frames):
            m.set_current(d, c)
            normals[k] = m.get_image(0, 1, 0)
    vmap = torch.empty((K.height, K.width, 4), dtype=torch.float32, device="cuda")
    st = dict(kind="fuse", m=m, frames=frames, normals=normals, poses=[sc.pose(k) for k in range(n)], play=_Player(n),
              vmap=vmap, nmap=torch.empty_like(vmap))
    for _ in range(n):
        _run_fuse(st)
    return st


def _prepare_track(case, seed):
    K = _intrinsics(case["width"], case["height"])
    n = 4
    sc = L.SynthScene(seed=seed)
    frames = [(_metres(d), c) for d, c in _frames(sc, K, range(n))]
    m = L.DenseTracking(K, _config(0.01, "ref", case["levels"], blocks=1 << 12))
    return dict(kind="track", m=m, frames=frames, play=_Player(n))


def _prepare_view(case, seed):
    K = _intrinsics(case["width"], case["height"])
    sc = _large_room(seed)
    m = L.DenseMapping(K, _config(case["voxel"], case["layout"], blocks=1 << 18))
    for k in range(0, 6 * case["frames"], 6):
        d, c = sc.render(K, k)
        m.update(_metres(d), c, sc.pose(k))
    n, poses = 12, []
    for k in range(n):  # the operator's camera swings 20 degrees to each side of the path
        a = 0.35 * math.sin(2.0 * math.pi * k / n)
        turn = np.eye(4)
        turn[0, 0], turn[0, 2], turn[2, 0], turn[2, 2] = math.cos(a), math.sin(a), -math.sin(a), math.cos(a)
        poses.append(sc.pose(6 * k % (6 * case["frames"])) @ turn)
    vmap = torch.empty((K.height, K.width, 4), dtype=torch.float32, device="cuda")
    return dict(kind="view", m=m, poses=poses, play=_Player(n), vmap=vmap, nmap=torch.empty_like(vmap),
                rgb=torch.empty((K.height, K.width, 3), dtype=torch.uint8, device="cuda"))


def _scan_blocks(case, seed):
    """At least `blocks` blocks of a scanned room, in an order of their own: coords, sdf, weight, rgb."""
    K = _intrinsics(640, 480)
    sc = L.SynthScene(seed=seed)
    m = L.DenseMapping(K, _config(case["voxel"], case["layout"], blocks=1 << 18))
    k = 0
    while k < 600 and m.stats().allocated_blocks < case["blocks"]:
        for j in (k, k + 2, k + 4):  # three looks from nearly the same place, then on along the loop
            d, c = sc.render(K, j)
            m.update(_metres(d), c, sc.pose(j))
        k += 30
    coords, sdf, w, rgb = m.export()
    order = np.lexsort((coords[:, 2], coords[:, 1], coords[:, 0]))[:case["blocks"]]
    return coords[order], sdf[order], w[order], rgb[order]


def _prepare_mesh(case, seed):
    coords, sdf, w, rgb = _scan_blocks(case, seed)
    # A session holding these blocks in this order: triangles come out in pool
    # order, which a whole frame's blocks get from a race, so each block is
    # allocated by an update of its own (one valid pixel, one block deep) before
    # the voxels are imported.
    voxel = case["voxel"]
    n = len(coords)
    K = L.IntrinsicMatrix(64, 64, 64.0, 64.0, 32.0, 32.0)
    m = L.DenseMapping(K, _config(voxel, case["layout"], blocks=max(1024, 1 << (n - 1).bit_length()), truncation=4 * voxel,
                                  zmin_update=0.9, zmax_update=1.1))
    depth = torch.zeros((64, 64), dtype=torch.float32, device="cuda")
    depth[32, 32] = 1.0
    grey = torch.zeros((64, 64, 3), dtype=torch.uint8, device="cuda")
    T = np.eye(4)
    for at in (coords.astype(np.float64) + 0.5) * (8.0 * voxel):
        T[:3, 3] = at
        T[2, 3] -= 1.0
        m.update(depth, grey, T)
    m.import_blocks(coords, sdf, w, rgb)
    most = 160 * n  # a scanned room meshes to about 90 triangles a block
    vertex = torch.zeros((most, 3, 3), dtype=torch.float32, device="cuda")
    attr = torch.zeros((most, 3, 3), dtype=torch.uint8 if case["mode"] == "colour" else torch.float32, device="cuda")
    return dict(kind="mesh", m=m, mode=case["mode"], vertex=vertex, attr=attr)


def _prepare_park(case, seed):
    K = _intrinsics(case["width"], case["height"])
    sc = L.SynthScene(seed=seed)
    n = 8
    cfg = _config(case["voxel"], case["layout"], blocks=1 << 16)
    pair = [L.System(K, cfg), L.System(K, cfg)]
    pair[0].set_pose(sc.pose(0))
    frames = _frames(sc, K, range(n))
    play = _Player(n)
    for _ in range(n):
        d, c = frames[play.next()]
        pair[0].process_images(d, c)
    host = torch.empty(2 * pair[0].snapshot_bytes(), dtype=torch.uint8, pin_memory=True)
    return dict(kind="park", pair=pair, frames=frames, play=play, host=host)


_PREPARE = dict(frame=_prepare_frame, tick=_prepare_tick, fuse=_prepare_fuse, track=_prepare_track, view=_prepare_view,
                mesh=_prepare_mesh, park=_prepare_park)


# ------------------------------------------------------------------ run

def run(state):
    return _RUN[state["kind"]](state)


def _run_frame(st):
    s = st["s"]
    d, c = st["frames"][st["play"].next()]
    if st["host"]:
        s.stage(d, c)
        s.process_staged()
    else:
        s.process_images(d, c)
    return {"pose": s.get_camera_pose(), "preview": s.get_rendered_image()}


def _run_tick(st):
    st["b"].process(st["active"])
    _stage_tick(st)
    poses, tracked, status, index = st["b"].results()
    preview = st["sessions"][st["shown"]].get_rendered_image()
    st["shown"] = (st["shown"] + 1) % len(st["sessions"])
    return {"poses": poses, "tracked": tracked, "status": status.astype(np.int64), "preview": preview}


def _run_fuse(st):
    k = st["play"].next()
    m, (d, c) = st["m"], st["frames"][k]
    m.update(d, c, st["poses"][k], normal=st["normals"][k])
    m.raycast(st["vmap"], st["poses"][k], nmap=st["nmap"])
    return {"vmap": st["vmap"], "nmap": st["nmap"]}


def _run_track(st):
    k = st["play"].next()
    m, f = st["m"], st["frames"]
    m.set_reference(*f[k])
    m.set_current(*f[k + 1 if k + 1 < len(f) else k - 1])
    r = m.compute_transform()
    return {"update": r.update, "icp_error": float(r.icp_error), "rgb_error": float(r.rgb_error)}


def _run_view(st):
    m, T = st["m"], st["poses"][st["play"].next()]
    m.raycast_check_visibility(st["vmap"], T)
    m.raycast(st["vmap"], T, nmap=st["nmap"], rgb=st["rgb"])
    return {"vmap": st["vmap"], "nmap": st["nmap"], "image": L.render_scene(st["vmap"], st["nmap"], st["rgb"])}


def _run_mesh(st):
    m, v, a = st["m"], st["vertex"], st["attr"]
    if st["mode"] == "vertex":
        return {"triangles": m.fetch_mesh_vertex_only(v), "vertex": v}
    n = m.fetch_mesh_with_normal(v, a) if st["mode"] == "normal" else m.fetch_mesh_with_colour(v, a)
    return {"triangles": n, "vertex": v, st["mode"]: a}


def _run_park(st):
    a, b = st["pair"]
    snap = a.snapshot(out=st["host"])
    b.restore(snap)
    at = b.get_camera_pose()[:3, 3]
    b.prune_async(center=at, radius=3.0)
    b.process_images(*st["frames"][st["play"].next()])
    st["pair"] = [b, a]
    return {"pose": b.get_camera_pose(), "preview": b.get_rendered_image()}


_RUN = dict(frame=_run_frame, tick=_run_tick, fuse=_run_fuse, track=_run_track, view=_run_view, mesh=_run_mesh,
            park=_run_park)


# ------------------------------------------------------------------ work

def _iterations(P, levels):
    """Pixel-iterations of the 10 / 5 / 3 / 3 schedule."""
    return sum(it * (P >> (2 * l)) for l, it in enumerate([10, 5, 3, 3, 3][:levels]))


def _pyramid(P, levels):
    return sum(P >> (2 * l) for l in range(levels))


def _visible(voxel):
    """Blocks of 8 voxels in view: about 35 m2 of block faces per look into a room."""
    return 35.0 / (8.0 * voxel) ** 2


def _bytes_per_voxel(layout):
    return 12 if layout == "ref" else 8


def _frame_work(P, voxel, layout, levels):
    v = _visible(voxel)
    # the frame in, each visible voxel read and written, the model prediction (vertices and normals) of the last
    # frame in and of this one out
    return (5 * P + 2 * _bytes_per_voxel(layout) * 512 * v + 64 * _pyramid(P, levels),
            230 * _iterations(P, levels) + 60 * 512 * v + 2000 * P)


def work(case):
    kind = case["kind"]
    if kind == "mesh":
        n = case["blocks"]
        out = 36 + (36 if case["mode"] == "normal" else 9 if case["mode"] == "colour" else 0)
        size = 8 if case["layout"] == "ref" else 4
        tris = 90 * n
        return {"bytes": n * 512 * (size + (4 if case["mode"] == "colour" else 0)) + tris * out,
                "flops": n * 512 * 20 + tris * 60}
    P = case["width"] * case["height"]
    if kind == "frame":
        b, f = _frame_work(P, case["voxel"], case["layout"], case["levels"])
        return {"bytes": b + 36 * P, "flops": f}
    if kind == "tick":
        each = [_frame_work(P, v, case["layout"], 3) for v in (0.005, 0.006, 0.008, 0.010)]
        n = case["sessions"] / 4.0
        return {"bytes": n * sum(b for b, _ in each) + 36 * P, "flops": n * sum(f for _, f in each)}
    if kind == "track":
        return {"bytes": 2 * 7 * P + 128, "flops": 230 * _iterations(P, case["levels"]) + 400 * P}
    v, s = _visible(case["voxel"]), _bytes_per_voxel(case["layout"])
    if kind == "fuse":
        return {"bytes": (7 + (16 if case["normals"] else 0)) * P + 2 * s * 512 * v + 32 * P,
                "flops": 60 * 512 * v + 2000 * P}
    if kind == "view":  # the voxels near the surface in view once, the maps and the image out
        return {"bytes": 0.25 * s * 512 * v + 39 * P, "flops": 4000 * P}
    b, f = _frame_work(P, case["voxel"], case["layout"], 3)
    snap = 1.6 * v * (s * 512 + 21) + 36 * _pyramid(P, 3)
    return {"bytes": b + 4 * snap + 36 * P, "flops": f}


# ------------------------------------------------------------------ exact

def exact(case, seed):
    """The odometry in 64 bits.  The other kinds return maps of hits: which voxel
    stops a ray, and so which pixels are set at all, hangs on the rounding of the
    stored voxels, and meshes on their order and table, so they have no such value."""
    if case["kind"] != "track":
        return None
    K = _intrinsics(case["width"], case["height"])
    sc = L.SynthScene(seed=seed)
    f = [(_metres(d), c) for d, c in _frames(sc, K, range(2))]
    ref = _pyramid64(f[0], K, case["levels"])
    cur = _pyramid64(f[1], K, case["levels"])
    T = torch.eye(4, dtype=torch.float64, device="cuda")
    prev = T.clone()
    err = [math.inf, math.inf]
    for level in reversed(range(case["levels"])):
        std, counts, last = 0.0, [0, 0], [math.inf, math.inf]
        for _ in range([10, 5, 3, 3, 3][level]):
            (A, b, res_i, n_i), (B, c, res_r, n_r) = _rows64(ref[level], cur[level], T, std)
            xi = torch.linalg.solve(1e6 * A + B, 1e6 * b + c)
            prev, T = T, _exp64(xi) @ T
            std = math.sqrt(res_r / (n_r - 6))
            now = [math.sqrt(res_i) / n_i, math.sqrt(res_r) / n_r]
            stop = False
            for q in (0, 1):
                if now[q] > last[q]:
                    if counts[q] >= 2:
                        T, stop = prev, True
                        break
                    counts[q] += 1
                    now[q] = last[q]
                else:
                    counts[q] = 0
                last[q] = err[q] = now[q]
            if stop:
                break
    return {"update": torch.linalg.inv(T), "icp_error": None, "rgb_error": None}


def _pyramid64(frame, K, levels):
    """Depth and intensity pyramids, vertices, normals and gradients of a frame."""
    d, c = frame[0].double(), frame[1].double()
    pad = torch.nn.functional.pad
    grey = 0.299 * c[..., 0] + 0.587 * c[..., 1] + 0.114 * c[..., 2]
    H, W = d.shape
    e = pad(d[None, None], (2, 2, 2, 2), mode="reflect")[0, 0]
    s1 = s2 = 0.0
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            if dx * dx + dy * dy <= 4:
                v = e[2 + dy:2 + dy + H, 2 + dx:2 + dx + W]
                w = torch.exp(-0.5 * (dx * dx + dy * dy) - 0.5 * (v - d) ** 2)
                s1, s2 = s1 + w * v, s2 + w
    d = s1 / s2
    got = []
    fx, fy, cx, cy = K.fx, K.fy, K.cx, K.cy
    for level in range(levels):
        if level:
            d = 0.25 * (d[0::2, 0::2] + d[0::2, 1::2] + d[1::2, 0::2] + d[1::2, 1::2])
            k = torch.tensor([1.0, 4.0, 6.0, 4.0, 1.0], dtype=torch.float64, device=d.device) / 16.0
            g = pad(grey[None, None], (2, 2, 2, 2), mode="reflect")
            g = torch.nn.functional.conv2d(g, k.view(1, 1, 1, 5))
            grey = torch.nn.functional.conv2d(g, k.view(1, 1, 5, 1))[0, 0][::2, ::2]
            fx, fy, cx, cy = 0.5 * fx, 0.5 * fy, 0.5 * cx, 0.5 * cy
        H, W = d.shape
        y, x = torch.meshgrid(torch.arange(H, dtype=torch.float64, device=d.device),
                              torch.arange(W, dtype=torch.float64, device=d.device), indexing="ij")
        z = torch.where((d > 0.3) & (d < 5.0), d, torch.full_like(d, math.nan))
        v = torch.stack([z * (x - cx) / fx, z * (y - cy) / fy, z], -1)

        def diff(a):
            left = torch.cat([a[:, :1], a[:, :-1]], 1)
            up = torch.cat([a[:1], a[:-1]], 0)
            return a.roll(-1, 1) - left, a.roll(-1, 0) - up

        a, b = diff(v)
        n = torch.linalg.cross(a, b)
        n = n / n.norm(dim=-1, keepdim=True)
        gx, gy = (0.5 * t for t in diff(grey))
        n[-1], n[:, -1] = math.nan, math.nan
        for t in (gx, gy):
            t[-1], t[:, -1] = 0.0, 0.0
        got.append(dict(v=v, n=n, i=grey, gx=gx, gy=gy, K=(fx, fy, cx, cy)))
    return got


def _normal_equations(rows, res, weight):
    r, e = rows * weight[:, None], res * weight
    return r.T @ r, r.T @ e, float((e * e).sum()), int(len(e))


def _rows64(ref, cur, T, std):
    """Point-to-plane and photometric normal equations at T: (A, b, squared residual, rows) of each."""
    H, W = ref["i"].shape
    fx, fy, cx, cy = ref["K"]
    p = ref["v"].reshape(-1, 3) @ T[:3, :3].T + T[:3, 3]
    n = ref["n"].reshape(-1, 3) @ T[:3, :3].T
    u = torch.floor(p[:, 0] / p[:, 2] * fx + cx + 0.5)
    v = torch.floor(p[:, 1] / p[:, 2] * fy + cy + 0.5)
    q = torch.nonzero((u >= 0) & (v >= 0) & (u < W) & (v < H))[:, 0]
    at = (v[q] * W + u[q]).long()
    vc, nc = cur["v"].reshape(-1, 3)[at], cur["n"].reshape(-1, 3)[at]
    ok = ((torch.linalg.cross(nc, n[q]).norm(dim=-1) < math.cos(30 * 3.14 / 180))
          & ((p[q] - vc).norm(dim=-1) <= 0.01) & ~nc.isnan().any(-1) & ~n[q].isnan().any(-1))
    q, vc = q[ok], vc[ok]
    icp = _normal_equations(torch.cat([n[q], torch.linalg.cross(p[q], n[q])], -1), ((vc - p[q]) * n[q]).sum(-1),
                            torch.ones(len(q), dtype=torch.float64, device=p.device))

    u, v = p[:, 0] / p[:, 2] * fx + cx, p[:, 1] / p[:, 2] * fy + cy
    q = torch.nonzero((u >= 2) & (u < W - 2) & (v >= 2) & (v < H - 2))[:, 0]
    u, v, p = u[q], v[q], p[q]
    x, y = u.floor().long(), v.floor().long()
    a, b = u - x, v - y

    def tap(img):
        return (img[y, x] * (1 - a) + img[y, x + 1] * a) * (1 - b) + (img[y + 1, x] * (1 - a) + img[y + 1, x + 1] * a) * b

    gx, gy, res = tap(cur["gx"]), tap(cur["gy"]), tap(cur["i"]) - ref["i"].reshape(-1)[q]
    ok = (gx > 2) | (gy > 2)
    gx, gy, res, p = gx[ok], gy[ok], res[ok], p[ok]
    if std > 10e-5:
        res = res / std
    w = torch.ones_like(res)
    if std > 10e-6:
        far = res.abs() > 1.345 * std
        w[far] = torch.sqrt(1.345 * std / res[far].abs())
    lx, ly = gx * fx / p[:, 2], gy * fy / p[:, 2]
    g = torch.stack([lx, ly, -(lx * p[:, 0] + ly * p[:, 1]) / p[:, 2]], -1)
    rgb = _normal_equations(torch.cat([g, torch.linalg.cross(p, g)], -1), -res, w)
    return icp, rgb


def _exp64(xi):
    """SE(3) exponential, translation first."""
    M = torch.zeros((4, 4), dtype=torch.float64, device=xi.device)
    M[0, 1], M[0, 2], M[1, 2] = -xi[5], xi[4], -xi[3]
    M[1, 0], M[2, 0], M[2, 1] = xi[5], -xi[4], xi[3]
    M[:3, 3] = xi[:3]
    return torch.linalg.matrix_exp(M)
