"""The Gauss-Newton step's solve, exponential and composition (csrc/gn_step.cuh)
against exact rational arithmetic."""
import ctypes as C
import subprocess
from fractions import Fraction as F
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent
EPS = 2.0 ** -52


@pytest.fixture(scope="module")
def step(tmp_path_factory):
    from libfusion_gb300 import build as B
    exe = tmp_path_factory.mktemp("gn") / "gn_step"
    subprocess.run([B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "-fmad=false", str(HERE / "gn_step_main.cu"), "-o",
                    str(exe)], check=True, capture_output=True)

    def run(A, b, T):
        low = np.tril_indices(6)
        rows = np.concatenate([A[:, low[0], low[1]], b, T.reshape(len(A), 12)], 1).astype(np.float64)
        r = subprocess.run([str(exe)], input=rows.tobytes(), capture_output=True, check=True)
        o = np.frombuffer(r.stdout).reshape(len(A), 18)
        return o[:, :6], o[:, 6:].reshape(-1, 3, 4)
    return run


def solve_exact(A, b):
    """Gaussian elimination in rationals; unknowns of all-zero rows are zero."""
    live = [i for i in range(6) if any(A[i])]
    M = [[F(float(A[i][j])) for j in live] + [F(float(b[i]))] for i in live]
    n = len(live)
    for k in range(n):
        p = max(range(k, n), key=lambda i: abs(M[i][k]))
        M[k], M[p] = M[p], M[k]
        for i in range(n):
            if i != k and M[i][k]:
                f = M[i][k] / M[k][k]
                M[i] = [x - f * y for x, y in zip(M[i], M[k])]
    x = [0.0] * 6
    for k, i in enumerate(live):
        x[i] = float(M[k][n] / M[k][k])
    return np.array(x)


def exp_exact(x):
    """exp of the twist, translation first, by its series in rationals (40 terms: below 1e-20 for angles to 3)."""
    r, w = [F(float(v)) for v in x[:3]], [F(float(v)) for v in x[3:]]
    M = [[F(0), -w[2], w[1], r[0]], [w[2], F(0), -w[0], r[1]], [-w[1], w[0], F(0), r[2]], [F(0)] * 4]
    total = [[F(int(i == j)) for j in range(4)] for i in range(4)]
    term = [row[:] for row in total]
    one = F(1, 1 << 200)
    for k in range(1, 40):
        term = [[sum(term[i][q] * M[q][j] for q in range(4)) / k for j in range(4)] for i in range(4)]
        term = [[F(int(v / one)) * one for v in row] for row in term]  # 200 bits are enough
        total = [[a + b for a, b in zip(s, t)] for s, t in zip(total, term)]
    return total


@pytest.mark.parametrize("kind", ["random", "zeros", "tied", "diagonal", "large_angle", "tiny"])
def test_step_matches_exact_arithmetic(step, kind):
    rng = np.random.default_rng(3)
    n = 24
    A, b, T = np.zeros((n, 6, 6)), np.zeros((n, 6)), np.zeros((n, 3, 4))
    for i in range(n):
        Q, _ = np.linalg.qr(rng.normal(size=(6, 6)))
        d = 10.0 ** rng.uniform(0, 1 + i % 8, 6)
        A[i] = (Q * d) @ Q.T * 1e6
        if kind == "zeros":  # unknowns without any observation
            gone = rng.permutation(6)[:1 + i % 6]
            A[i][gone] = 0.0
            A[i][:, gone] = 0.0
        elif kind == "tied":  # equal diagonals: the tie in the pivot search
            A[i] = 4.0 * np.eye(6) + (np.ones((6, 6)) - np.eye(6)) * (1 + i % 3) / 4.0
        elif kind == "diagonal":
            A[i] = np.diag(2.0 ** rng.integers(-60, 60, 6).astype(np.float64))
        A[i] = np.tril(A[i]) + np.tril(A[i], -1).T
        x = rng.normal(size=6) * {"large_angle": 0.7, "tiny": 1e-9}.get(kind, 0.01)
        b[i] = A[i] @ x
        U, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        T[i, :, :3], T[i, :, 3] = U, rng.normal(size=3)
    xs, Ts = step(A, b, T)
    for i in range(n):
        live = A[i].any(0)
        cond = np.linalg.cond(A[i][np.ix_(live, live)]) if live.any() and kind != "diagonal" else 1.0
        want = solve_exact(A[i], b[i])
        # elimination with diagonal pivoting of a positive definite matrix: a backward error of
        # a few n eps in a normwise sense, amplified by the condition number
        assert np.linalg.norm(xs[i] - want) <= 40 * EPS * cond * np.linalg.norm(want) + 1e-300
        E = exp_exact(xs[i])
        for r in range(3):
            for c in range(4):
                exact = sum(E[r][k] * F(float(T[i, k, c])) for k in range(3)) + (E[r][3] if c == 3 else 0)
                # coefficients to a few eps (the closed forms above 1/4 rad lose another 2 / 0.0625)
                assert abs(float(exact - F(float(Ts[i, r, c])))) <= 80 * EPS * (1 + np.abs(T[i]).max())


def test_step_with_infinities_ends(step):
    A = np.tile(np.eye(6), (3, 1, 1))
    A[1, 2, 2], A[2, 4, 4] = np.inf, np.nan
    x, T = step(A, np.ones((3, 6)), np.tile(np.eye(3, 4), (3, 1, 1)))
    assert np.array_equal(x[0], np.ones(6))
    assert np.array_equal(x[1], [1, 1, 0, 1, 1, 1])  # b / infinity
    assert np.isnan(x[2]).any()


@pytest.mark.parametrize("gate", ["dist", "angle"])
def test_icp_gates_at_their_thresholds(gbf, gate):
    """sine < angle and dist <= dist_max hold for the rounded square roots: thresholds
    at, next below and next above the roots of pixels, zero, negative, tiny, huge,
    infinite and NaN ones count the pixels that the comparison of the roots counts."""
    import torch
    L = gbf
    w, h = 64, 16
    f = np.float32
    rng = np.random.default_rng(3)
    py, px = np.mgrid[0:h, 0:w].astype(f)
    ref = np.stack([px, py, np.ones_like(px), np.ones_like(px)], -1)  # fx = z = 1: pixel (x, y)
    cur, nr, nc = ref.copy(), np.zeros_like(ref), np.zeros_like(ref)
    cur[..., :3] += rng.normal(0, 10.0 ** rng.uniform(-4, 3, (h, w, 1)), (h, w, 3)).astype(f)
    nr[..., :3], nc[..., :3] = rng.normal(size=(2, h, w, 3)).astype(f) * f(0.6)
    cur[0, :8], nc[0, :8] = ref[0, :8], nr[0, :8]  # roots of zero
    a, b = nc, nr
    cr = [a[..., i] * b[..., j] - a[..., j] * b[..., i] for i, j in ((1, 2), (2, 0), (0, 1))]
    dd = [ref[..., i] - cur[..., i] for i in range(3)]
    dist, sine = (np.sqrt((v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]).ravel() for v in (dd, cr))
    assert dist.dtype == f and sine.dtype == f
    grey = np.full((h, w), 50, f)
    imgs = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (ref, nr, grey, cur, nc, grey, 0 * grey, 0 * grey)]
    roots = dist if gate == "dist" else sine
    picks = roots[rng.integers(0, roots.size, 24)]
    tests = np.concatenate([picks, np.nextafter(picks, f(0)), np.nextafter(picks, f(np.inf)),
                            np.array([0, -0.0, -1, 1e-45, 1e-30, 1e-20, 1e30, np.inf, np.nan], f)])
    out = torch.empty(58, dtype=torch.float64, device="cuda")
    for t in tests:
        d_max, angle = (t, f(np.inf)) if gate == "dist" else (f(np.inf), t)
        inp = L._lib.ReduceInputs(w, h, 1.0, 1.0, 0.0, 0.0, *[x.data_ptr() for x in imgs], float(d_max), float(angle))
        L._lib.call("gbf_reduce_noalloc", C.byref(inp), L._lib.mat16(np.eye(4)), 0.0, out.data_ptr(),
                    torch.cuda.current_stream().cuda_stream)
        want = np.count_nonzero((sine < angle) & (dist <= d_max))
        assert int(out.cpu()[28]) == want, (gate, t)
