"""Inside and distance queries on meshes whose faces differ in size, and at small counts.

The parity test reads a mesh's faces from crossing grids whose cells follow the mean edge unless
some faces are far larger, and the answers are the oracle's whatever the cells: parities exactly,
f32 distances bit for bit.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(lo, hi):
    c = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], float)
    f = np.array([[0, 1, 3], [0, 3, 2], [4, 6, 7], [4, 7, 5], [0, 4, 5], [0, 5, 1],
                  [2, 3, 7], [2, 7, 6], [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3]])
    return np.asarray(lo) + c * (np.asarray(hi) - np.asarray(lo)), f


def _ball(n, radius, bump):
    """A bumpy sphere of 4 n^2 - 4 n faces."""
    u, w = np.meshgrid(np.arange(2 * n) * np.pi / n, np.arange(1, n) * np.pi / n)
    r = radius * (1.0 + bump * np.sin(5 * u) * np.sin(3 * w))
    v = np.stack([r * np.sin(w) * np.cos(u), r * np.sin(w) * np.sin(u), r * np.cos(w)], -1)
    v = np.vstack([v.reshape(-1, 3), [0, 0, radius], [0, 0, -radius]])
    f, m, top = [], 2 * n, (n - 1) * 2 * n
    for i in range(m):
        j = (i + 1) % m
        f += [[top, i, j], [top + 1, (n - 2) * m + j, (n - 2) * m + i]]
        for k in range(n - 2):
            a, b, c, d = k * m + i, k * m + j, (k + 1) * m + i, (k + 1) * m + j
            f += [[a, c, b], [b, c, d]]
    return v, np.array(f)


def _join(*parts):
    vs, fs, at = [], [], 0
    for v, f in parts:
        vs.append(v)
        fs.append(f + at)
        at += len(v)
    return np.vstack(vs), np.vstack(fs)


MESHES = {
    "one_leaf": lambda: (_box([-1, -1, -1], [1, 1, 1])[0], _box([-1, -1, -1], [1, 1, 1])[1][:3]),
    "box": lambda: _box([-9, -8, -7], [9, 8, 7]),
    "ball": lambda: _ball(24, 9.0, 0.15),
    # Twelve faces a hundred mean edges across around a fine ball.
    "ball_in_box": lambda: _join(_ball(32, 0.9, 0.1), _box([-12, -11, -10], [12, 11, 10])),
    # Ten times as long as wide, and padding (1e-5 of the coordinates) above a cell.
    "far_needle": lambda: (_ball(16, 1.0, 0.0)[0] * [20, 2, 2] + [3e4, 0, 0], _ball(16, 1.0, 0.0)[1]),
}


@pytest.mark.parametrize("name", sorted(MESHES))
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 5000])
def test_queries_are_bit_exact(gpu_ctx, oracle, name, n):
    v, f = MESHES[name]()
    rng = np.random.default_rng(n)
    mid, half = (v.min(0) + v.max(0)) / 2, (v.max(0) - v.min(0)) / 2
    pts = mid + rng.uniform(-1.1, 1.1, size=(n, 3)) * half
    pts[::7] = v[rng.integers(0, len(v), size=len(pts[::7]))]  # on the surface
    g, c = gpu_ctx.mesh(v, f), oracle.Mesh(v, f)
    pose = np.eye(4)
    d_g, in_g = gpu_ctx.inside(g, pts, pose)
    d_c, in_c = c.inside(pts, pose)
    assert np.array_equal(in_g, in_c)
    assert np.array_equal(np.asarray(d_g).view(np.uint32), np.asarray(d_c).view(np.uint32))
    for window in (0.0, float(0.05 * half.min()), float(half.max()), np.inf):
        assert np.array_equal(gpu_ctx.bounded_distance(g, pts, pose, window),
                              c.bounded_distance(pts, pose, window)), window


def _soup(n, large):
    """n loose faces, `large` of them of about sixty times the others' size."""
    rng = np.random.default_rng(n)
    size = np.where(np.arange(n) < large, 3.0, 0.05)[:, None, None]
    v = rng.uniform(-10, 10, size=(n, 1, 3)) + rng.normal(size=(n, 3, 3)) * size
    return v.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3)


@pytest.mark.parametrize("n,large", [(1, 1), (31, 3), (33, 32), (257, 5), (3001, 30)])
def test_parities_among_faces_of_any_size(gpu_ctx, oracle, n, large):
    """Faces of one cell and of thousands side by side in a warp of the grids' build."""
    v, f = _soup(n, large)
    q = np.random.default_rng(n + 1).uniform(-12, 12, size=(5000, 3))
    gd, gi = gpu_ctx.inside(gpu_ctx.mesh(v, f), q, np.eye(4))
    cd, ci = oracle.Mesh(v, f).inside(q, np.eye(4))
    assert np.array_equal(gi, ci)
    assert np.array_equal(np.asarray(gd).view(np.uint32), np.asarray(cd).view(np.uint32))


def test_a_few_large_faces_do_not_hold_up_a_mesh(gpu_ctx):
    """A mesh with one large face in a hundred is built in the time of one without, and not in
    that of a thread that goes through the largest face's cells (seven times as long)."""
    import time

    def build(v, f):
        best = np.inf
        for _ in range(8):
            t0 = time.perf_counter()
            mesh = gpu_ctx.mesh(v, f)
            best = min(best, time.perf_counter() - t0)
            del mesh
        return best
    v, f = _soup(20000, 0)
    assert build(*_soup(20000, 200)) < 3.0 * build(v, f)
