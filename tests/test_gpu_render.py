"""The "next" rows around the per-frame path: a raycast from an arbitrary pose
with its own visibility pass (DenseMapping::raycast_check_visibility,
src/voxel_hashing/voxel_hashing.cpp:121-135) and headless Phong shading
(renderScene / renderSceneTextured, src/tracking/cuda_imgproc.cu:17-108), both
against the oracle."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _oracle_map(L, cfg, K):
    import oracle as O
    return O.OracleMap(O.config_from(cfg), O.intrinsics_from(K))


@pytest.mark.parametrize("layout", [0, 1, 2])
def test_raycast_check_visibility_bit_exact(gbf, layout):
    """Fuse along the trajectory, then raycast from a pose the last fuse did not
    see from: the visible list is rebuilt for that pose on both sides."""
    import torch
    L = gbf
    K = H.intrinsics(L)
    cfg = H.small_config(L, layout)
    m = L.DenseMapping(K, cfg)
    om = _oracle_map(L, cfg, K)
    fr = H.frames(L, K, 6, step=5)
    for d, c, T in fr:
        dm = H.depth_m(d)
        m.update(H.cuda(dm), H.cuda(c), T)
        om.fuse(dm, c, T)
    for T in (fr[1][2], fr[3][2]):
        vm = torch.full((K.height, K.width, 4), float("nan"), device="cuda")
        m.raycast_check_visibility(vm, T)
        g = vm.cpu().numpy()
        o = om.raycast_check_visibility(T)
        vg = {tuple(x) for x in m.visible_blocks()}
        vo = {tuple(x) for x in om.visible()}
        assert vg == vo, f"visible sets differ: {len(vg ^ vo)} blocks"
        assert np.array_equal(m.zrange(), om.zrange()), "z-range grids differ"
        gh, oh = ~np.isnan(g[..., 2]), ~np.isnan(o[..., 2])
        assert np.array_equal(gh, oh), f"hit masks differ in {np.sum(gh != oh)} pixels"
        assert gh.mean() > 0.8
        assert np.array_equal(g[gh], o[oh])


def _device_pow20(x):
    """CUDA's powf(x, 20.f) of float32 arguments (a float32 tensor-tensor pow)."""
    import torch
    t = torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()
    return torch.pow(t, torch.full_like(t, 20.0)).cpu().numpy()


def test_render_scene_matches_oracle(gbf):
    """Shaded model prediction of a System session, plain and textured, bit for
    bit: every step rounds as written on both sides, and the oracle takes
    CUDA's powf(x, 20) for the bases it evaluates (recorded in a first run).
    With libm's powf instead, a truncated 8-bit value may move by one on rare
    pixels, which the second check bounds."""
    import oracle as O
    import torch
    L = gbf
    K = H.intrinsics(L)
    s = L.System(K, H.small_config(L, 0))
    fr = H.frames(L, K, 3, step=3)
    s.set_pose(fr[0][2])
    for d, c, _ in fr:
        s.process_images(H.cuda(d), H.cuda(c))
    torch.cuda.synchronize()
    vm = s.get_image(1, 0, 0)  # model prediction: vertex / normal maps of the reference set
    nm = s.get_image(1, 1, 0)
    v, n = vm.cpu().numpy(), nm.cpu().numpy()
    assert np.isfinite(v[..., 2]).mean() > 0.8
    rgb = fr[-1][1]
    for textured in (False, True):
        g = (s.get_rendered_scene_textured() if textured else s.get_rendered_image()).cpu().numpy()
        exact, sizes, misses = O.with_device_transcendentals(
            lambda: O.render_scene(v, n, rgb if textured else None), {O.TRANS_POW20: _device_pow20})
        assert sizes[O.TRANS_POW20] > 1000 and misses[O.TRANS_POW20] == 0
        assert np.array_equal(g, exact)
        o = O.render_scene(v, n, rgb if textured else None)
        diff = np.abs(g.astype(np.int32) - o.astype(np.int32))
        assert diff.max() <= 1
        assert (diff > 0).mean() < 2e-3
        assert (g[..., 3] == 255).all()
        # the free function on the same maps gives the session's image
        f = L.render_scene(vm, nm, H.cuda(rgb) if textured else None).cpu().numpy()
        assert np.array_equal(f, g)
    # background colour where the prediction is empty
    bg = np.isnan(v[..., 0])
    if bg.any():
        assert (g[bg][:, :3] == O.render_scene(np.full((1, 1, 4), np.nan, np.float32),
                                               np.zeros((1, 1, 4), np.float32))[0, 0, :3]).all()


@pytest.mark.parametrize("voxel,zmin,far", [(0.01, 0.3, 0.0), (0.04, 0.05, 0.0), (0.004, 0.3, 0.0), (0.01, 0.3, 3000.0)])
def test_raycast_skips_only_empty_space(gbf, voxel, zmin, far):
    """Rays pass depth slices without a block unread and take neighbouring blocks
    from lists: from poses inside, at and away from the surfaces, with blocks that
    reach the camera plane, and with a map whose coordinates round a ray's steps
    (3 km from the origin: 1/64 voxel per step), vertices and hit masks are the
    oracle's bit for bit."""
    import oracle as O
    import torch
    L = gbf
    K = L.IntrinsicMatrix(168, 120, 110.0, 105.0, 80.3, 61.7)
    cfg = H.small_config(L, 0, voxel_size=voxel, truncation=3 * voxel, zmin_raycast=zmin, zmin_update=0.3,
                         num_blocks=1 << 16, num_buckets=1 << 18)
    m, om = L.DenseMapping(K, cfg), O.OracleMap(O.config_from(cfg), O.intrinsics_from(K))
    shift = np.array([far, -far, far / 2])
    poses = []
    for d, c, T in H.frames(L, K, 3, step=40, seed=5):
        T = T.copy()
        T[:3, 3] += shift
        m.update(H.cuda(H.depth_m(d)), H.cuda(c), T)
        om.fuse(H.depth_m(d), c, T)
        poses.append((T, H.depth_m(d)[60, 84]))
    rng = np.random.default_rng(2)
    vmap = torch.empty((K.height, K.width, 4), dtype=torch.float32, device="cuda")
    hits = 0
    for T, z in poses:
        for ahead in (0.0, 0.6 * z, z - 0.2, z, z + 0.05):  # up to and through the surface
            P = T.copy()
            a, b = rng.uniform(-0.6, 0.6, 2)
            R = np.array([[np.cos(a), 0, np.sin(a)], [0, 1, 0], [-np.sin(a), 0, np.cos(a)]]) @ \
                np.array([[np.cos(b), -np.sin(b), 0], [np.sin(b), np.cos(b), 0], [0, 0, 1]])
            P[:3, 3] += ahead * T[:3, 2]
            P[:3, :3] = T[:3, :3] @ R
            m.raycast_check_visibility(vmap, P)
            o = om.raycast_check_visibility(P)
            g = vmap.cpu().numpy()
            gh, oh = ~np.isnan(g[..., 2]), ~np.isnan(o[..., 2])
            assert np.array_equal(gh, oh) and np.array_equal(g[gh], o[oh])
            hits += int(gh.sum())
    assert hits > 5000


@pytest.mark.parametrize("before", ["new", "pruned", "restored"])
def test_raycast_refined_samples_before_the_near_plane(gbf, before):
    """A wall three voxels nearer than zmin_raycast, a block face between the two: a ray's
    first sample lies behind the wall and its refined one up to a truncation before
    the near plane, in a block that no marched sample can meet.  Vertices and hit masks are
    the oracle's on a new session's first raycast, after a prune that moved block
    ids, and after a restore into an arena that held another map."""
    import oracle as O
    import torch
    L = gbf
    K = L.IntrinsicMatrix(168, 120, 110.0, 105.0, 80.3, 61.7)
    cfg = H.small_config(L, 0, truncation=0.05, zmin_update=0.2, num_blocks=1 << 14, num_buckets=1 << 16)
    rgb = np.full((K.height, K.width, 3), 99, np.uint8)
    T = np.eye(4)
    T[2, 3] = 0.035  # block faces at depths 0.205 and 0.285
    aside, back = T.copy(), T.copy()
    aside[0, 3] = 20.0
    back[2, 3] -= 1.0
    vmap = torch.empty((K.height, K.width, 4), dtype=torch.float32, device="cuda")

    def fuse(m, z, P, n=3):
        for _ in range(n):
            m.update(torch.full((K.height, K.width), z, device="cuda"), H.cuda(rgb), P)
    m = L.System(K, cfg)
    if before == "pruned":
        fuse(m, 1.5, aside)
    fuse(m, 0.27, T)
    om = _oracle_map(L, cfg, K)
    for _ in range(3):
        om.fuse(np.full((K.height, K.width), 0.27, np.float32), rgb, T)
    if before == "pruned":
        m.raycast_check_visibility(vmap, back)  # every block's neighbours, by the ids before
        assert m.prune(center=[0, 0, 0], radius=5.0) > 100
    if before == "restored":
        snap = m.snapshot()
        m = L.System(K, cfg)
        fuse(m, 1.2, T)
        m.raycast_check_visibility(vmap, T)
        m.restore(snap)
    for dz in (0.0, 0.003, -0.004):
        P = T.copy()
        P[2, 3] += dz
        m.raycast_check_visibility(vmap, P)
        g, o = vmap.cpu().numpy(), om.raycast_check_visibility(P)
        gh, oh = ~np.isnan(g[..., 2]), ~np.isnan(o[..., 2])
        assert oh.mean() > 0.8 and np.nanmax(o[..., 2]) < cfg.zmin_raycast
        assert np.array_equal(gh, oh), f"hit masks differ in {np.sum(gh != oh)} pixels"
        assert np.array_equal(g[gh], o[oh])


def test_raycast_of_an_imported_map_beyond_the_truncation(gbf):
    """An imported map may hold any sdf.  Four times the sdf at a quarter of the truncation
    is the same surface: where a ray's first sample is not interpolated (sdf < -1/2) it is
    refined to the same point, two truncations before the near plane, with the same
    neighbours around it, whatever raycasts came before."""
    import torch
    L = gbf
    K = L.IntrinsicMatrix(168, 120, 110.0, 105.0, 80.3, 61.7)
    cfg = [H.small_config(L, L.VOXEL_HALF, truncation=t, zmin_update=0.2, num_blocks=1 << 14, num_buckets=1 << 16)
           for t in (0.0625, 0.015625)]
    rgb = np.full((K.height, K.width, 3), 99, np.uint8)
    T = np.eye(4)
    T[2, 3] = 0.035  # block faces at depths 0.205 and 0.285
    a, b = (L.DenseMapping(K, c) for c in cfg)
    a.update(torch.full((K.height, K.width), 0.259, device="cuda"), H.cuda(rgb), T)
    coords, sdf, w, col = a.export()
    b.import_blocks(coords, 4 * sdf, w, col)
    out = [torch.empty((K.height, K.width, 4), dtype=torch.float32, device="cuda") for _ in range(2)]
    for m, v in zip((a, b), out):
        m.raycast_check_visibility(v, T)
    g, h = (v.cpu().numpy() for v in out)
    hit = ~np.isnan(g[..., 2])
    assert hit.mean() > 0.8 and np.nanmax(g[..., 2]) < cfg[0].zmin_raycast
    assert np.array_equal(g, h, equal_nan=True), f"differ in {np.sum(hit != ~np.isnan(h[..., 2]))} hits"


def test_update_keeps_the_last_raycasts_zrange(gbf):
    """The z-range grid and the renderable count are the last raycast's until the next one:
    an update in between makes neither."""
    import torch
    L = gbf
    K = H.intrinsics(L)
    m = L.DenseMapping(K, H.small_config(L, 2))
    fr = H.frames(L, K, 2, step=10)
    vmap = torch.empty((K.height, K.width, 4), dtype=torch.float32, device="cuda")
    m.update(H.cuda(H.depth_m(fr[0][0])), H.cuda(fr[0][1]), fr[0][2])
    m.raycast(vmap, fr[0][2])
    grid, count = m.zrange(), m.stats().render_blocks_valid
    assert count > 100 and grid.max() > 0.3
    m.update(H.cuda(H.depth_m(fr[1][0])), H.cuda(fr[1][1]), fr[1][2])
    assert m.stats().render_blocks_valid == count and np.array_equal(m.zrange(), grid)
