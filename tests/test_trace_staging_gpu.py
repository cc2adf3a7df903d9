"""Traces over host buffers against the device call (closest hits to the bit, any hit whether there is one:
which occluder a query reports is left open): at the edges of the staging units (4096
rays) and chunks (32768), with fewer and more chunks than there are slots (4), from pageable, pinned and
mixed buffers, and with the hits written over the rays."""
import ctypes as C

import numpy as np
import pytest
import torch

from liar_b200 import trace as T

pytestmark = pytest.mark.gpu

CHUNK = 32768


def _mesh(ctx):
    rng = np.random.default_rng(3)
    c = rng.random((3000, 1, 3)) * 2 - 1
    v = (c + 0.1 * (rng.random((3000, 3, 3)) - 0.5)).reshape(-1, 3).astype(np.float32)
    return T.Mesh(ctx, v, np.arange(9000, dtype=np.uint32).reshape(-1, 3))


def _rays(n):
    rng = np.random.default_rng(n)
    r = np.empty((n, 8), np.float32)
    r[:, 0:3] = rng.random((n, 3)) * 3 - 1.5
    r[:, 3] = 0
    r[:, 4:7] = rng.normal(size=(n, 3))
    r[:, 7] = np.inf
    return r


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("n", [1, 4095, 4097, CHUNK, CHUNK + 1, 4 * CHUNK, 4 * CHUNK + 1, 8 * CHUNK, 8 * CHUNK + 1, 27 * CHUNK + 4099])
def test_host_buffers_match_the_device_call(n, any_hit):
    ctx = T.Context()
    mesh, rays = _mesh(ctx), _rays(n)
    unstaged = mesh.intersect(rays, any_hit=any_hit)
    mesh.intersect(_rays(1 << 20))  # from as many rays on, calls are staged
    d = torch.from_numpy(rays).cuda()
    out = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    mesh.trace_into(d.data_ptr(), n, out.data_ptr(), any_hit=any_hit)
    ctx.synchronize()
    ref = out.cpu().numpy()

    def check(prim, t):
        if any_hit:
            np.testing.assert_array_equal(prim >= 0, ref[:, 0] >= 0)
        else:
            np.testing.assert_array_equal(prim, ref[:, 0])
            np.testing.assert_array_equal(t.view(np.int32), ref[:, 1])

    check(*unstaged)
    for _ in range(2):  # the second call finds the slots and events of the first
        check(*mesh.intersect(rays, any_hit=any_hit))
    pinned_in, pinned_out = torch.from_numpy(rays).pin_memory(), torch.empty((n, 2), dtype=torch.int32).pin_memory()
    over = rays.copy()
    for src, dst in ((rays, np.empty((n, 2), np.int32)), (rays, pinned_out.numpy()),
                     (pinned_in.numpy(), np.empty((n, 2), np.int32)), (pinned_in.numpy(), pinned_out.numpy()), (over, over)):
        if dst is not over:
            dst.fill(-7)
        ctx.check(ctx._lib.liar_gpu_trace(ctx.handle, mesh.handle, C.c_void_p(src.ctypes.data), n,
                                          C.c_void_p(dst.ctypes.data), int(any_hit)))
        hits = dst.view(np.int32).ravel()[:2 * n].reshape(n, 2)
        check(hits[:, 0], np.ascontiguousarray(hits[:, 1]))
