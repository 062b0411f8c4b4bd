"""The ICP rung gives the same bytes whatever block and cluster shape it runs at.

A rung runs on a 256-thread block, a 512-thread block or a cluster of 2, 4 or 8 of those per
start, by the number of starts and source points, and keeps matches from pass to pass without
searching for them again. Its sums have one order for all of these, so a start's registration is
one set of bytes; the poses are the oracle's within the ICP tests' own bounds (1e-6 t and 1e-4
degrees).
"""

from __future__ import annotations

import numpy as np
import pytest

from _slab import origin_t, trace_deg

pytestmark = pytest.mark.gpu

T = 10.0
STARTS = (1, 18, 19, 37, 38, 74, 75, 296, 297)  # the edges of the forms on 148 SMs


def _surface(rng, n):
    """n points of a wavy sheet with their unit normals."""
    uv = rng.uniform(-30.0, 30.0, size=(n, 2))
    z = 3.0 * np.sin(uv[:, 0] / 6.0) + 2.0 * np.cos(uv[:, 1] / 5.0)
    g = np.stack([-0.5 * np.cos(uv[:, 0] / 6.0), 0.4 * np.sin(uv[:, 1] / 5.0), np.ones(n)], 1)
    return np.column_stack([uv, z]), g / np.linalg.norm(g, axis=1, keepdims=True)


def _starts(rng, k):
    from importlib import import_module
    synth = import_module("sherd-refit_b200.synth")
    out = np.empty((k, 4, 4))
    for i in range(k):
        step = rng.normal(size=3) * 0.03 * T
        out[i] = synth.rigid(synth.random_rotation(rng, 2.0), step)
    return out


@pytest.mark.parametrize("estimation", [1, 0], ids=["plane", "point"])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 511, 512, 1023, 1024, 2047, 2048, 4321])
def test_a_start_is_registered_alike_in_every_form(gpu_ctx, oracle, n, estimation):
    rng = np.random.default_rng(n)
    tp, tn = _surface(rng, 3000)
    src, _ = _surface(rng, n)
    target = gpu_ctx.cloud(tp, tn)
    starts = _starts(rng, max(STARTS))
    dist = 0.2 * T
    regs = {k: gpu_ctx.icp_rung_array(src, target, starts[:k], dist, 12, estimation=estimation)
            for k in STARTS}
    for k in STARTS:
        assert regs[k].tobytes() == regs[max(STARTS)][:k].tobytes(), k
    ref = oracle.icp_rung(src, oracle.Cloud(tp, tn), starts[:4], dist, 12,
                          point_to_point=estimation == 0)
    if n >= 257:  # fewer points may leave the normal equations near singular
        for g, r in zip(regs[max(STARTS)], ref):
            pose = g["transform"].reshape(4, 4)
            want = np.array(r.transform[:]).reshape(4, 4)
            assert origin_t(pose, want, T) < 1e-6 and trace_deg(pose, want) < 1e-4
            assert int(g["correspondences"]) == r.correspondences


@pytest.mark.parametrize("estimation", [1, 0], ids=["plane", "point"])
@pytest.mark.parametrize("n", [20_011, 200_001])
def test_large_sources_are_registered_alike_in_every_form(gpu_ctx, n, estimation):
    """Long passes, in which the blocks of a cluster drift apart: none may write its matches while
    another still sums over them."""
    rng = np.random.default_rng(n)
    tp, tn = _surface(rng, 3000)
    src, _ = _surface(rng, n)
    target = gpu_ctx.cloud(tp, tn)
    starts = _starts(rng, 297)
    whole = gpu_ctx.icp_rung_array(src, target, starts, 0.2 * T, 12, estimation=estimation)
    for k in (1, 18, 37, 74) * 3:
        some = gpu_ctx.icp_rung_array(src, target, starts[:k], 0.2 * T, 12, estimation=estimation)
        assert some.tobytes() == whole[:k].tobytes(), k


@pytest.mark.parametrize("distance", [1e-3, 0.5, 40.0, 1e4])
def test_radii_from_no_match_to_every_point(gpu_ctx, oracle, distance):
    rng = np.random.default_rng(5)
    tp, tn = _surface(rng, 1500)
    src, _ = _surface(rng, 900)
    starts = _starts(rng, 80)
    starts[1, :3, 3] += 500.0  # far from the target: no match at the smaller radii
    target = gpu_ctx.cloud(tp, tn)
    few = gpu_ctx.icp_rung_array(src, target, starts[:2], distance, 8)
    many = gpu_ctx.icp_rung_array(src, target, np.tile(starts, (4, 1, 1)), distance, 8)
    assert few.tobytes() == many[:2].tobytes()
    assert many[:80].tobytes() == many[240:].tobytes()
    ref = oracle.icp_rung(src, oracle.Cloud(tp, tn), starts[:2], distance, 0)
    first = gpu_ctx.icp_rung_array(src, target, starts[:2], distance, 0)
    for g, r in zip(first, ref):  # one pass: the matches themselves
        assert int(g["correspondences"]) == r.correspondences


def test_targets_above_16_bits_and_batches_of_every_form(sherd, gpu_ctx, gpu_slab, slab):
    """One pair's items in one batch, and the same items pair by pair: the same candidates for
    every number of items, with 16-bit and 32-bit match slots."""
    rng = np.random.default_rng(9)
    tp, tn = _surface(rng, 66000)
    big = gpu_ctx.cloud(tp, tn)
    src, _ = _surface(rng, 700)
    a, b = gpu_slab["a"]["surf"], gpu_slab["b"]["surf"]
    wide = gpu_ctx.pair(a, b, big, gpu_slab["frac_t"], src, src[:300], gpu_slab["scales"])
    starts = _starts(rng, 6)
    for pair, inits in ((wide, starts), (gpu_slab["pair"], slab["starts"].reshape(-1, 4, 4))):
        whole = None
        for n in (1, 40, 100, 300):
            items = [(0, k, inits[k % len(inits)]) for k in range(n)]
            got = gpu_ctx.ladder_verify_batch([pair], items, sherd.default_params())
            cands = sherd.candidates(got)[:n]
            first = cands["rungs"][:1].tobytes() + cands["scores"][:1].tobytes()
            whole = whole or first
            assert first == whole, n
        plain = sherd.candidates(gpu_ctx.ladder_verify_batch([pair], items[:40],
                                                             sherd.default_params(), sherd.SCHED_PLAIN))
        assert plain.tobytes() == cands[:40].tobytes()


@pytest.mark.parametrize("limit", [0.0, 0.3], ids=["plain_ladder", "early_rejection"])
@pytest.mark.parametrize("n", [300, 600, 1100, 2100])
def test_ladders_run_alike_in_every_form(sherd, gpu_ctx, gpu_slab, slab, n, limit):
    """The queue's items shared by a cluster's blocks, in one launch or split by the early
    rejection: the same candidates on clusters of 8, 4 and 2 blocks, on wide blocks and on narrow
    ones, under both schedules."""
    b = gpu_slab["b"]["arrays"]  # its clouds, cut or repeated to n and n / 2 points
    pair = gpu_ctx.pair(gpu_slab["a"]["surf"], gpu_slab["b"]["surf"], gpu_slab["reg_t"],
                        gpu_slab["frac_t"], np.resize(b["reg_p"], (n, 3)),
                        np.resize(b["frac_p"], (n // 2, 3)), gpu_slab["scales"])
    inits = slab["starts"].reshape(-1, 4, 4)
    params = sherd.default_params()
    params.early_reject_tight = limit

    def run(k, sched):
        items = [(0, i, inits[i % len(inits)]) for i in range(k)]
        return sherd.candidates(gpu_ctx.ladder_verify_batch([pair], items, params, sched)).copy()
    whole = run(max(STARTS), sherd.SCHED_BATCHED)
    partial = int(whole["scores"]["partial"].sum())
    assert 0 < partial < len(whole) if limit else partial == 0
    for k in STARTS * 2:
        for sched in (sherd.SCHED_BATCHED, sherd.SCHED_PLAIN):
            assert run(k, sched).tobytes() == whole[:k].tobytes(), (k, sched)
