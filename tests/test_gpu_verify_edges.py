"""Verification at the edges of its launch shapes: few and odd sample counts, meshes of one leaf,
poses with nothing inside, and batches around the size where the scores run side by side.

Every score is the oracle's, bit for bit, as in the fixture's verification test.
"""

from __future__ import annotations

import threading

import numpy as np
import pytest

from _slab import SCORE_KEYS
from test_gpu_queries import _ball, _box

pytestmark = pytest.mark.gpu


def _side(lib, mesh, rng, n_f, n_s, n_b):
    v, f = mesh
    m = lib.mesh(v, f) if hasattr(lib, "mesh") else lib.Mesh(v, f)
    half = max(1, len(f) // 2)
    frac = m.subset((np.arange(len(f)) < half).astype(np.uint8))

    def on(n, faces):
        tri = v[f[rng.integers(0, faces, size=n)]]
        w = rng.dirichlet(np.ones(3), size=n)
        e = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
        return (tri * w[:, :, None]).sum(1), e / np.linalg.norm(e, axis=1, keepdims=True)
    pf, s = on(n_f, half)[0], on(n_s, len(f))[0]
    bp, bn = on(n_b, half)
    mp, mn = on(n_b, len(f))
    make = lib.surfaces if hasattr(lib, "surfaces") else lib.Surfaces
    return make(frac, m, 1, 50.0, pf, s, bp, bn, mp, mn)


def _pose(angle, shift):
    p = np.eye(4)
    c, s = np.cos(angle), np.sin(angle)
    p[:2, :2] = [[c, -s], [s, c]]
    p[:3, 3] = shift
    return p


MESHES = {"ball": lambda: _ball(16, 9.0, 0.1), "box": lambda: _box([-8, -7, -6], [8, 7, 6]),
          "flat": lambda: (np.array([[-9, -9, 0], [9, -9, 0], [9, 9, 1], [-9, 9, 0.]]),
                           np.array([[0, 1, 2], [0, 2, 3]]))}


@pytest.mark.parametrize("a,b", [("ball", "ball"), ("ball", "box"), ("box", "flat")])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 65, 1023, 1025])
def test_scores_are_the_oracles_at_every_count(gpu_ctx, gpu_slab, oracle, slab, a, b, n):
    scales = oracle.scales_from(slab["scales"])
    t = gpu_slab["scales"].t
    g = [_side(gpu_ctx, MESHES[k](), np.random.default_rng(n + i), n, n, n) for i, k in
         enumerate((a, b))]
    c = [_side(oracle, MESHES[k](), np.random.default_rng(n + i), n, n, n) for i, k in
         enumerate((a, b))]
    # Deep inside one another, overlapping, nothing inside but near, and far away.
    for pose in (_pose(0.3, [0.1, 0.2, 0.3]), _pose(0.1, [8, 0, 2]), _pose(0.7, [22.0 + 0.1 * t, 0, 0]),
                 _pose(0.0, [900, -700, 800])):
        sg = gpu_ctx.verify(g[0], g[1], pose, gpu_slab["scales"])
        sc = oracle.verify(c[0], c[1], pose, scales)
        for key in SCORE_KEYS:
            assert np.array_equal(getattr(sg, key), getattr(sc, key), equal_nan=True), (key, pose)


def test_candidates_do_not_depend_on_the_batch_size(sherd, gpu_ctx, gpu_slab, slab):
    """1 to 74 items score side by side, more of them an item a block, on 148 SMs."""
    starts = slab["starts"]
    params = sherd.default_params()
    sizes = (1, 18, 19, 37, 73, 74, 75, 76, 149, 296, 300)
    got = {}
    for n in sizes:
        items = [(0, k, starts[k % len(starts)]) for k in range(n)]
        got[n] = sherd.candidates(gpu_ctx.ladder_verify_batch([gpu_slab["pair"]], items, params)).copy()
    for n in sizes:
        assert got[n].tobytes() == got[sizes[-1]][:n].tobytes(), n


@pytest.mark.parametrize("far", [3e4, 3e6, 4e7, 5e17])
def test_scores_of_runaway_poses_are_the_oracles(gpu_ctx, gpu_slab, oracle, slab, far):
    """Poses at which f32 merges points, and then faces: the least distance is still exact."""
    scales = oracle.scales_from(slab["scales"])
    g, c = ([_side(lib, MESHES["ball"](), np.random.default_rng(i), 500, 2000, 70) for i in (1, 2)]
            for lib in (gpu_ctx, oracle))
    pose = _pose(0.4, [far, -0.3 * far, 0.1 * far])
    sg = gpu_ctx.verify(g[0], g[1], pose, gpu_slab["scales"])
    sc = oracle.verify(c[0], c[1], pose, scales)
    for key in SCORE_KEYS:
        assert np.array_equal(getattr(sg, key), getattr(sc, key), equal_nan=True), key


def test_one_pose_holds_scratch_for_one_pose(sherd, gpu_slab, slab):
    """Device memory goes by the items of a call, not by what the device could run at once: at
    10^6 samples a side one item takes four score blocks' scratch of 4 MB each (444 blocks' would
    be 1.8 GB), and a ladder of two items two slots of 200,000 points (592 slots' would be 1 GB).
    """
    import torch

    ctx = sherd.Context(0)
    n = 1_000_000
    a, b = (_side(ctx, MESHES["ball"](), np.random.default_rng(i), n, 5000, 70) for i in (1, 2))
    rng = np.random.default_rng(3)
    src = rng.normal(size=(200_000, 3))
    tgt = rng.normal(size=(500, 3))
    cloud = ctx.cloud(tgt, tgt / np.linalg.norm(tgt, axis=1, keepdims=True))
    pair = ctx.pair(a, b, cloud, cloud, src, src, gpu_slab["scales"])
    pose = _pose(0.3, [0.1, 0.2, 0.3])

    def held(call):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        call()
        return before - torch.cuda.mem_get_info()[0]
    assert held(lambda: ctx.verify(a, b, pose, gpu_slab["scales"])) < 200 << 20
    items = [(0, k, pose) for k in range(2)]
    for sched in (sherd.SCHED_BATCHED, sherd.SCHED_PLAIN):
        for limit in (0.0, 0.3):
            params = sherd.default_params()
            params.early_reject_tight = limit
            assert held(lambda: ctx.ladder_verify_batch([pair], items, params, sched)) < 200 << 20


def test_an_aborted_ladder_is_not_verified(sherd, gpu_slab):
    """A batch small enough for its scores to go side by side, aborted while its ladder runs, does
    not begin them: the verification stage takes next to nothing of its own time."""
    ctx = sherd.Context(0)
    n = 500_000
    a, b = (_side(ctx, MESHES["ball"](), np.random.default_rng(i), n, 500, 70) for i in (1, 2))
    rng = np.random.default_rng(3)
    src, tgt = rng.normal(size=(400_000, 3)), rng.normal(size=(5000, 3))
    cloud = ctx.cloud(tgt, tgt / np.linalg.norm(tgt, axis=1, keepdims=True))
    pair = ctx.pair(a, b, cloud, cloud, src, src, gpu_slab["scales"])
    items = [(0, k, _pose(0.01 * k, [0.1, 0.2, 0.3])) for k in range(70)]
    batch = ctx.batch([pair], items, sherd.default_params())
    whole = batch.run()
    assert whole["ladder"] > 100.0  # milliseconds: the abort below comes while it runs
    stop = threading.Timer(0.02, ctx.abort)
    ms = np.zeros(len(batch.STAGES), np.float32)
    stop.start()
    code = sherd.lib().sherd_batch_run(batch.h, ms)
    stop.join()
    assert code == -4
    assert ms[1] < 0.2 * whole["verify"], (whole, ms)
    assert batch.run().keys() == whole.keys()
