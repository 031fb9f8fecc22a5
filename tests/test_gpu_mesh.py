"""Marching cubes over blocks of made-up voxels against a plain restatement:
values and weights at the thresholds, missing neighbours, several chunks of the
offset scan, and a buffer that ends within a block."""
import re
from pathlib import Path

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
EDGES = [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7)]
TABLE = [int(x, 16) for x in re.findall(r"0x[0-9a-f]+", (Path(__file__).parents[1] / "oracle/mc_table.inc").read_text())]


def _cluster(side, n, noisy, rng):
    """n blocks of a side^3 cube; `noisy` of them random with special values, the rest +1."""
    c = np.stack(np.meshgrid(*[np.arange(side) - side // 2] * 3, indexing="ij"), -1).reshape(-1, 3)
    c = c[rng.permutation(len(c))[:n]].astype(np.int32)
    sdf, w = np.ones((n, 512), np.float32), np.ones((n, 512), np.float32)
    special = np.array([0.0, 2.0 ** -24, -2.0 ** -24, 16 * 2.0 ** -24, 17 * 2.0 ** -24, -16 * 2.0 ** -24, -17 * 2.0 ** -24],
                       np.float32)  # fp16 values on both sides of 1e-6
    weights = np.array([0.0, 0.0009994507, 0.0010004044, 1.0, 255.0], np.float32)  # fp16 values around 1e-3
    for i in rng.permutation(n)[:noisy]:
        v = rng.uniform(-1, 1, 512).astype(np.float16).astype(np.float32)
        v[:64] = special[rng.integers(0, len(special), 64)]
        sdf[i] = v[rng.permutation(512)]
        w[i] = weights[rng.choice(len(weights), 512, p=[0.02, 0.01, 0.01, 0.9, 0.06])]
    return c, sdf, w, rng.integers(0, 256, (n, 512, 3), dtype=np.uint8)


def _mesh(c, sdf, w, rgb, mode, voxel):
    f = np.float32
    at = {tuple(x): i for i, x in enumerate(c)}
    tris, attrs = [], []
    for b, pos in enumerate(c):
        S, ok, col = np.zeros((9, 9, 9), f), np.zeros((9, 9, 9), bool), np.zeros((9, 9, 9, 3), np.uint8)
        for d in np.ndindex(2, 2, 2):  # z, y, x
            i = at.get((pos[0] + d[2], pos[1] + d[1], pos[2] + d[0]))
            if i is None:
                continue
            dst = tuple(slice(8, 9) if k else slice(0, 8) for k in d)
            src = tuple(slice(0, 1) if k else slice(0, 8) for k in d)
            S[dst] = sdf[i].reshape(8, 8, 8)[src]
            wi = w[i].reshape(8, 8, 8)[src]
            ok[dst] = wi.astype(np.float64) > 1e-3 if mode == 2 else wi != 0
            col[dst] = rgb[i].reshape(8, 8, 8, 3)[src]
        if not (S < 0).any():
            continue
        for z, y, x in np.ndindex(8, 8, 8):
            s = [S[z + dz, y + dy, x + dx] for dx, dy, dz in CORNERS]
            if not all(ok[z + dz, y + dy, x + dx] for dx, dy, dz in CORNERS):
                continue
            packed = TABLE[sum(1 << k for k in range(8) if s[k] < 0)]
            for t in range(packed & 15):
                tri, colour = [], []
                for q in range(3):
                    e = packed >> (4 + 12 * t + 4 * q) & 15
                    a, bb = s[EDGES[e][0]], s[EDGES[e][1]]
                    val = f(0) if abs(float(a)) < 1e-6 else f(1) if abs(float(bb)) < 1e-6 else \
                        f(0) if abs(float(a - bb)) < 1e-6 else (f(0) - a) / (bb - a)
                    off = [(val, 0, 0), (1, val, 0), (f(1) - val, 1, 0), (0, f(1) - val, 0)][e & 3] if e < 8 else \
                        (*CORNERS[e - 8][:2], val)
                    off = (off[0], off[1], f(e >= 4)) if e < 8 else off
                    tri.append([(f(pos[k] * 8 + (x, y, z)[k]) + f(off[k])) * voxel for k in range(3)])
                    dx, dy, dz = CORNERS[e if e < 8 else e - 8]
                    colour.append(col[z + dz, y + dy, x + dx])
                tris.append(tri)
                attrs.append(colour)
    return np.array(tris, f), np.array(attrs, np.uint8)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("pool", [4096, 1 << 19])  # chunks of 1,024 and of 2,048 blocks
def test_mesh_of_made_up_blocks(gbf, pool, mode):
    import torch
    L = gbf
    c, sdf, w, rgb = _cluster(13, 2100, 24, np.random.default_rng(mode))
    m = L.DenseMapping(H.intrinsics(L, 64, 64), H.small_config(L, 1, num_blocks=pool, num_buckets=1 << 20))
    m.import_blocks(c, sdf, w, rgb)
    want, colours = _mesh(c, sdf, w, rgb, mode, np.float32(0.01))
    cap = len(want) + 5
    vtx = torch.full((cap, 3, 3), 7.0, dtype=torch.float32, device="cuda")
    attr = torch.full((cap, 3, 3), 7, dtype=torch.uint8 if mode == 2 else torch.float32, device="cuda")
    fetch = [lambda v, a: m.fetch_mesh_vertex_only(v), m.fetch_mesh_with_normal, m.fetch_mesh_with_colour][mode]
    assert fetch(vtx, attr) == len(want) and len(want) > 5000
    v, a = vtx.cpu().numpy(), attr.cpu().numpy()
    assert np.all(v[len(want):] == 7) and np.all(a[len(want):] == 7)  # nothing past the end
    extra = [a[:len(want)]] if mode == 2 else []
    got, ref = H.sort_tris(v[:len(want)], *extra), H.sort_tris(want, *([colours] if mode == 2 else []))
    for x, y in zip(got, ref):
        assert np.array_equal(x, y)
    if mode == 1:
        n = a[:len(want)].astype(np.float64)
        e = v[:len(want)].astype(np.float64)
        cr = np.cross(e[:, 1] - e[:, 0], e[:, 2] - e[:, 0])
        good = np.linalg.norm(cr, axis=1) > 1e-6
        cr = cr[good] / np.linalg.norm(cr[good], axis=1, keepdims=True)
        # coordinates to 0.5 m in float: differences of millimetres carry 3e-5, a unit normal of a
        # triangle of 1e-6 m2 and edges to 1.4 cm then at most a few 1e-3
        assert np.abs(n[good] - cr[:, None, :]).max() < 5e-3
        assert np.array_equal(a[:len(want), 0], a[:len(want), 1], equal_nan=True)
        assert np.array_equal(a[:len(want), 0], a[:len(want), 2], equal_nan=True)
    # a buffer that ends within a block: the same triangles, cut
    short = torch.full((cap, 3, 3), 7.0, dtype=torch.float32, device="cuda")
    k = len(want) // 2 + 3
    assert fetch(short[:k], attr) == k
    s = short.cpu().numpy()
    assert np.array_equal(s[:k], v[:k]) and np.all(s[k:] == 7)
