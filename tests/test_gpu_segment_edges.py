"""Segmentation and breaklines where their kernels change over: balls too large for a warp and for
a block's first size, and breaklines longer than the room a first call brings."""

from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from test_gpu_queries import _ball
from test_gpu_segment import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,thick", [(16, 2.0), (48, 16.0), (64, 80.0)],
                         ids=["warp", "block", "large_block"])
def test_balls_of_every_size_are_bit_exact(gpu_ctx, oracle, n, thick):
    """A face's ball of radius thick / 4 holds up to about 25, 600 and 16,000 faces."""
    v, f = _ball(n, 9.0, 0.05)
    res = float(np.linalg.norm(v[f[:, 0]] - v[f[:, 1]], axis=1).mean())
    gpu = gpu_ctx.segment(gpu_ctx.mesh(v, f), v, f, thick, res, trace=True)
    cpu = oracle.segment(oracle.Mesh(v, f), v, f, thick, res)
    _compare(gpu, cpu)


def test_balls_of_different_sizes_on_two_threads(sherd):
    """Two threads with a context each, one of whose balls need more shared memory: both get the
    labels they get alone."""
    jobs = []
    for n, thick in ((48, 16.0), (64, 80.0)):
        ctx = sherd.Context(0)
        v, f = _ball(n, 9.0, 0.05)
        res = float(np.linalg.norm(v[f[:, 0]] - v[f[:, 1]], axis=1).mean())
        mesh = ctx.mesh(v, f)
        jobs.append(lambda c=ctx, m=mesh, v=v, f=f, t=thick, r=res: c.segment(m, v, f, t, r))
    alone = [job()[0] for job in jobs]
    with ThreadPoolExecutor(2) as pool:
        both = [pool.submit(lambda job=job: [job()[0] for _ in range(60)])
                for job in jobs]
        for want, got in zip(alone, both):
            assert all(np.array_equal(want, g) for g in got.result())


@pytest.mark.parametrize("share", [0.0, 0.02, 0.5])
def test_breaklines_of_any_length_are_the_oracles(gpu_ctx, oracle, share):
    """Labels drawn face by face: none, a line within the first call's room, one beyond it."""
    v, f = _ball(48, 9.0, 0.05)
    frac = np.random.default_rng(5).random(len(f)) < share
    g = gpu_ctx.breaklines(v, f, frac, 2.0)
    c = oracle.breaklines(v, f, frac, 2.0)
    assert len(g["p"]) == len(c["p"])
    if share == 0.5:
        assert len(g["p"]) > 256 + 16 * int(len(f) ** 0.5)
    for k in ("p", "valid", "sub"):
        assert np.array_equal(g[k], c[k]), k
