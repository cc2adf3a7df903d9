"""The gather's selection of the k nearest at its edges: k around a warp's width and the list's end, many
photons at one distance or one place, queries on photons, fewer photons than k in reach, dense cells
beside sparse ones. Neighbours, their order (equal distances: lower index first) and distances are the
oracle's; the estimate agrees with a 64-bit sum over them for photon counts of every record alignment."""
import ctypes as C

import numpy as np
import pytest

import oracle
from liar_b200.photons import PhotonMap

pytestmark = pytest.mark.gpu


def cloud(kind):
    rng = np.random.default_rng(5)
    if kind == "spot":  # a dense spot on a sparse plane, and a lattice with many equal distances
        p = rng.uniform(-1, 1, (6000, 3))
        p[:, 1] = 0
        p[:2500] = p[:2500] * 0.02 + [0.3, 0, 0.1]
        q = np.concatenate([rng.uniform(-1, 1, (300, 3)) * [1, 0.01, 1], p[:100], p[3000:3100]])
        return p, q, 0.4
    if kind == "lattice":
        g = np.stack(np.meshgrid(*[np.arange(13.0)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.125
        q = np.concatenate([g[::7], g[::11] + 0.0625])
        return g[rng.permutation(len(g))], q, 0.6
    p = np.concatenate([np.zeros((700, 3)), np.full((90, 3), 0.25), rng.uniform(-0.5, 0.5, (400, 3))])
    return p[rng.permutation(len(p))], np.array([[0, 0, 0], [0.25, 0.25, 0.25], [0.1, 0, 0], [5, 5, 5], [0.2, 0.2, 0.26]]), 0.5


@pytest.mark.parametrize("kind", ["spot", "lattice", "piles"])
@pytest.mark.parametrize("k", [1, 2, 31, 32, 33, 50, 63, 64])
def test_neighbours_at_the_edges(gpu_ctx, kind, k):
    p, q, r = cloud(kind)
    p, q = p.astype(np.float32), q.astype(np.float32)
    idx, d2, cnt = PhotonMap(gpu_ctx, p, r_max=r).gather(q, k)
    ri, rd, rc = oracle.knn(p, q, k, r)
    np.testing.assert_array_equal(cnt, rc)
    np.testing.assert_array_equal(idx, ri)
    np.testing.assert_array_equal(d2[ri >= 0].view(np.int32), rd[ri >= 0].view(np.int32))


@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 33, 64])
@pytest.mark.parametrize("n, offset", [(64, 0), (65, 0), (67, 1), (66, 3)])
def test_estimate_sums_every_record(gpu_ctx, k, n, offset):
    """offset: floats past a 16-byte boundary at which the photon arrays start."""
    import torch
    g = torch.Generator().manual_seed(n)
    def photons():
        x = torch.zeros(3 * n + 8, device="cuda")
        x[offset:offset + 3 * n] = torch.randn(3 * n, generator=g).cuda()
        return x[offset:offset + 3 * n]
    power, omega = photons(), photons()
    nq = 37
    normals = torch.randn((nq, 3), generator=g).cuda()
    idx = torch.stack([torch.randperm(n, generator=g)[:k] if k <= n else torch.arange(k) % n for _ in range(nq)]).int().cuda()
    idx[0, 0], idx[1, 0] = n - 1, 0
    d2 = torch.rand((nq, k), generator=g).sort(1).values.cuda() + 0.1
    cnt = torch.randint(0, k + 1, (nq,), generator=g).int().cuda()
    out = torch.empty((nq, 3), device="cuda")
    torch.cuda.synchronize()
    gpu_ctx.check(gpu_ctx._lib.liar_gpu_photon_estimate_device(
        gpu_ctx.handle, power.data_ptr(), omega.data_ptr(), n, normals.data_ptr(), nq, k, idx.data_ptr(), d2.data_ptr(),
        cnt.data_ptr(), C.c_float(0.5), out.data_ptr(), None))
    gpu_ctx.synchronize()
    P, O, N, I = (x.cpu().double().numpy() for x in (power.view(-1, 3), omega.view(-1, 3), normals, idx))
    I = I.astype(int)
    c = cnt.cpu().numpy()
    use = (np.arange(k)[None] < c[:, None]) & ((O[I] * N[:, None]).sum(2) > 0)
    far = d2.cpu().double().numpy()[np.arange(nq), np.maximum(c, 1) - 1]
    ref = (P[I] * use[..., None]).sum(1) * np.where(c > 0, 0.5 / (np.pi * far), 0.0)[:, None]
    # rounding of up to 64 terms of about 1 and of the scale: 64 * 2^-24 of the sum of magnitudes
    bound = (np.abs(P[I]) * use[..., None]).sum(1) * np.where(c > 0, 0.5 / (np.pi * far), 0.0)[:, None] * 70 * 2.0 ** -24 + 1e-12
    assert np.all(np.abs(out.cpu().double().numpy() - ref) <= bound)


@pytest.mark.parametrize("n", [1, 3, 1023, 1024, 1025, 5000, 2_100_003])
@pytest.mark.parametrize("flat", [False, True], ids=["volume", "surface"])
def test_maps_of_every_size(gpu_ctx, n, flat):
    """Map builds below and above the density estimate's first size, with sampled photons in it, and over
    odd counts; a rebuild with fewer photons in the same buffers answers for those alone."""
    import torch
    rng = np.random.default_rng(n)
    p = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    if flat:
        p[:, 1] = 0.25
    q = np.concatenate([p[:: max(1, n // 150)][:150], rng.uniform(-1, 1, (50, 3)).astype(np.float32)])
    if flat:
        q[:, 1] = 0.25
    r = 1.5 * (60 / max(n, 60)) ** (1 / 2 if flat else 1 / 3)
    m = PhotonMap(gpu_ctx, p, r_max=r)
    for count in (n, (n + 1) // 2):
        if count != n:
            d = torch.from_numpy(p[:count]).cuda()
            torch.cuda.synchronize()
            m.rebuild(d.data_ptr(), count)
        idx, d2, cnt = m.gather(q, 33)
        ri, rd, rc = oracle.knn_grid(p[:count], q, 33, r)
        np.testing.assert_array_equal(cnt, rc)
        np.testing.assert_array_equal(idx, ri)
        np.testing.assert_array_equal(d2[ri >= 0].view(np.int32), rd[ri >= 0].view(np.int32))
