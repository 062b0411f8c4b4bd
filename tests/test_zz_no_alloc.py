"""The allocation-free ICP rung (sherd_icp_rung_noalloc) against sherd_icp_rung.

Some callers cannot allocate device memory in the middle of a run: a worker held to a device
memory budget fixed up front, or code that must not call cudaMalloc/cudaFree while other
streams are in flight, because both can block or synchronise the whole device. For them the
rung keeps its per-point working memory in one fixed array inside the library and takes inputs
and outputs that already live on the device. Here the test itself allocates those buffers
(with torch) and checks two calls in a row against the allocating entry point, within the
tolerance the other ICP tests use (1e-6 t and 1e-4 degrees on at least 8 of the 10 starts).
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from _slab import origin_t, piece, trace_deg

pytestmark = pytest.mark.gpu


def _call(sherd, ctx, src, n, target, inits, k, opt, out):
    return sherd.lib().sherd_icp_rung_noalloc(ctx.h, C.c_void_p(src), n, target.h,
                                              C.c_void_p(inits), k, opt, C.c_void_p(out))


@pytest.mark.parametrize("estimation", [1, 0], ids=["point_to_plane", "point_to_point"])
def test_the_allocation_free_rung_matches_the_allocating_one(sherd, gpu_ctx, slab, estimation):
    import torch

    a, b = piece(slab, "pieceA"), piece(slab, "pieceB")
    target = gpu_ctx.cloud(a["reg_p"], a["reg_n"])
    t, icp = float(slab["scales"][0]), float(slab["scales"][11])
    dist = 0.2 * t * icp
    starts = np.ascontiguousarray(slab["starts"].reshape(-1, 16))
    k, n = len(starts), len(b["reg_p"])
    expected = gpu_ctx.icp_rung(b["reg_p"], target, starts, dist, 30, estimation=estimation)

    src = np.zeros((n, 4))
    src[:, :3] = b["reg_p"]
    d_src = torch.from_numpy(src).cuda()
    d_inits = torch.from_numpy(starts.copy()).cuda()
    d_out = torch.empty(C.sizeof(sherd.Registration) * k, dtype=torch.uint8, device="cuda")
    opt = sherd.IcpOptions(estimation, 30, dist)
    calls = []
    for _ in range(2):
        d_out.fill_(0xFF)
        torch.cuda.synchronize()
        rc = _call(sherd, gpu_ctx, d_src.data_ptr(), n, target, d_inits.data_ptr(), k, opt,
                   d_out.data_ptr())
        assert rc == 0, sherd.lib().sherd_last_error(gpu_ctx.h)
        host = d_out.cpu().numpy().tobytes()
        calls.append((sherd.Registration * k).from_buffer_copy(host))

    for regs in calls:
        close = 0
        for got, want in zip(regs, expected):
            pg, pw = got.pose(), want.pose()
            if origin_t(pg, pw, t) < 1e-6 and trace_deg(pg, pw) < 1e-4:
                close += 1
                assert got.correspondences == want.correspondences
        assert close >= 8, close
    assert bytes(calls[0]) == bytes(calls[1])


def test_the_allocation_free_rung_refuses_what_it_cannot_hold(sherd, gpu_ctx, slab):
    import torch

    a, b = piece(slab, "pieceA"), piece(slab, "pieceB")
    target = gpu_ctx.cloud(a["reg_p"], a["reg_n"])
    n = len(b["reg_p"])
    d_src = torch.zeros((n, 4), dtype=torch.float64, device="cuda")
    d_inits = torch.zeros((1, 16), dtype=torch.float64, device="cuda")
    d_out = torch.empty(C.sizeof(sherd.Registration), dtype=torch.uint8, device="cuda")
    opt = sherd.IcpOptions(1, 30, 1.0)
    too_many = (1 << 20) // n + 1  # the capacity is k * n_source <= 2^20
    rc = _call(sherd, gpu_ctx, d_src.data_ptr(), n, target, d_inits.data_ptr(), too_many, opt,
               d_out.data_ptr())
    assert rc == -1
    assert b"SHERD_NOALLOC_CAPACITY" in sherd.lib().sherd_last_error(gpu_ctx.h)
    rc = _call(sherd, gpu_ctx, d_src.data_ptr() + 8, n, target, d_inits.data_ptr(), 1, opt,
               d_out.data_ptr())
    assert rc == -1
    # Misaligned poses or records, and host memory, are refused on the host before a launch.
    rc = _call(sherd, gpu_ctx, d_src.data_ptr(), n, target, d_inits.data_ptr() + 4, 1, opt,
               d_out.data_ptr())
    assert rc == -1 and b"aligned" in sherd.lib().sherd_last_error(gpu_ctx.h)
    rc = _call(sherd, gpu_ctx, d_src.data_ptr(), n, target, d_inits.data_ptr(), 1, opt,
               d_out.data_ptr() + 4)
    assert rc == -1 and b"aligned" in sherd.lib().sherd_last_error(gpu_ctx.h)
    host_inits = np.zeros(16)
    rc = _call(sherd, gpu_ctx, d_src.data_ptr(), n, target, host_inits.ctypes.data, 1, opt,
               d_out.data_ptr())
    assert rc == -1 and b"device" in sherd.lib().sherd_last_error(gpu_ctx.h)


FIRST_CALLS = """
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
from importlib import import_module
import numpy as np
import torch
sherd = import_module("sherd-refit_b200")
ctx = sherd.Context(0)
p = np.random.default_rng(0).normal(size=(3000, 3))
target = ctx.cloud(p, p / np.linalg.norm(p, axis=1, keepdims=True))
src = torch.zeros((4096, 4), dtype=torch.float64, device="cuda")
src[:, :3] = torch.from_numpy(np.random.default_rng(1).normal(size=(4096, 3)))
inits = torch.eye(4, dtype=torch.float64, device="cuda").reshape(1, 16).repeat(400, 1).contiguous()
out = torch.empty(C.sizeof(sherd.Registration) * 400, dtype=torch.uint8, device="cuda")
free = []
# The sizes by which a rung takes its blocks and clusters, on 148 SMs.
for k, n in ((400, 100), (100, 600), (60, 600), (30, 1100), (10, 4000)):
    rc = sherd.lib().sherd_icp_rung_noalloc(
        ctx.h, C.c_void_p(src.data_ptr()), n, target.h, C.c_void_p(inits.data_ptr()), k,
        sherd.IcpOptions(1, 3, 0.5), C.c_void_p(out.data_ptr()))
    assert rc == 0, sherd.lib().sherd_last_error(ctx.h)
    free.append(torch.cuda.mem_get_info()[0])
print(free)
assert len(set(free)) == 1, free
"""


def test_after_the_first_call_no_form_of_the_rung_takes_device_memory():
    """The rung runs on blocks and clusters by its size: a call of one form up front must do for
    all of them. In a process of its own, in which nothing has been loaded before."""
    import subprocess
    import sys
    from pathlib import Path

    run = subprocess.run([sys.executable, "-c", FIRST_CALLS, str(Path(__file__).resolve().parent.parent)],
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout + run.stderr
