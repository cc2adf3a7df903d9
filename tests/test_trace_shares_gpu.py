"""Launches of the trace kernels with few rays: a warp's share of the rays runs from one ray, traced by
the whole warp, over shares below a warp's width to full batches from the work counter. Hits are the
oracle's, index and bits of t, at each of these sizes and at the ends between them."""
import numpy as np
import pytest

import oracle
from liar_b200 import scenes
from liar_b200.trace import Mesh

pytestmark = pytest.mark.gpu

WARPS = 148 * 32  # resident warps of the launch shapes


@pytest.fixture(scope="module")
def shell():
    """A model with long rays along its surface, the rays of the largest size, and the oracle's hits."""
    v, f = scenes.displaced_icosphere(levels=6, seed=3)
    n = 33 * WARPS + 5
    r = scenes.random_rays(v, n, seed=11)
    r[::7, 3] = 0.1
    r[::5, 7] = 0.9
    r[::9, 3] = -0.5           # hits behind the origin count
    d = np.random.default_rng(0).normal(size=(n // 3, 3))
    d -= (d * r[: n // 3, :3]).sum(1, keepdims=True) * r[: n // 3, :3]
    r[: n // 3, :3] /= np.linalg.norm(r[: n // 3, :3], axis=1, keepdims=True)
    r[: n // 3, 4:7] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)  # tangent rays
    tree = oracle.Tree(v, f)
    return v, f, r, tree.trace(r), tree.trace(r, any_hit=True)


@pytest.mark.parametrize("shape", [(128, 16), (128, 8), (256, 8)], ids=str)
@pytest.mark.parametrize("leaf", [4, 8])
def test_every_share_gives_the_oracles_hits(gpu_ctx, shell, shape, leaf):
    v, f, rays, (p_ref, t_ref), (a_ref, _) = shell
    mesh = Mesh(gpu_ctx, v, f, max_leaf_size=leaf)
    saved = gpu_ctx.trace_config
    gpu_ctx.trace_config = shape
    try:
        for n in (1, 2, 31, 33, 1000, WARPS, WARPS + 1, 8 * WARPS, 8 * WARPS + 1, 9 * WARPS, 32 * WARPS, 33 * WARPS + 5):
            p, t = mesh.intersect(rays[:n])
            hit = p_ref[:n] >= 0
            np.testing.assert_array_equal(p, p_ref[:n], err_msg=f"{n} rays")
            np.testing.assert_array_equal(t[hit].view(np.int32), t_ref[:n][hit].view(np.int32), err_msg=f"{n} rays")
            a, _ = mesh.intersect(rays[:n], any_hit=True)
            np.testing.assert_array_equal(a >= 0, a_ref[:n] >= 0, err_msg=f"{n} rays, any hit")
    finally:
        gpu_ctx.trace_config = saved
        mesh.close()
