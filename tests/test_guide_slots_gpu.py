"""Network evaluation at the edges of its work split: tiles of 128 rows, dealt to one slot of every SM
before the second slot of any, six slots an SM. Rows do not depend on one another and every row runs the
same sequence of MMAs, so a row's mixture is the same bits whatever tile it falls into; the last rows are
compared with the oracle at the tolerances of the evaluation test."""
import numpy as np
import pytest
import torch

import oracle
from liar_b200 import guiding as GD
from liar_b200.kernel import default_context

pytestmark = pytest.mark.gpu

LO, HI = np.array([-1, -1, -1], np.float32), np.array([2, 1, 3], np.float32)


def _rows(tiles_per_sm, rest):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return tiles_per_sm * sms * 128 + rest


@pytest.mark.parametrize("tiles_per_sm, rest", [(0, 127), (0, 128), (0, 129), (1, -1), (1, 1), (5, 77), (6, -128), (6, 1), (13, 5)])
def test_rows_are_the_same_in_every_tile_and_slot(tiles_per_sm, rest):
    n = _rows(tiles_per_sm, rest)
    rng = np.random.default_rng(n)
    x = (np.concatenate([LO, [-1] * 6]) + rng.random((n, 9)) * np.concatenate([HI - LO, [2] * 6])).astype(np.float32)
    g = GD.Guide(default_context(), (LO, HI), seed=5)
    xg = torch.from_numpy(x).cuda()
    mix = g.eval(xg).cpu().numpy()
    sms = _rows(1, 0) // 128
    tiles = (n + 127) // 128
    for t in sorted({0, 1, sms - 1, sms, 5 * sms, 6 * sms - 1, 6 * sms, 12 * sms, tiles - 2, tiles - 1}):
        if not 0 <= t < tiles:
            continue
        lo, hi = t * 128, min(n, t * 128 + 128)
        # shifted by a row, so that each row is another thread's and tile's than before
        for a, b in ((lo, hi), (lo + 1, min(n, hi + 1))):
            if a < b:
                np.testing.assert_array_equal(g.eval(xg[a:b].clone()).cpu().numpy(), mix[a:b])
    m = min(n, 130)
    _, ref = oracle.guide_forward(g.params, x[-m:], LO, HI, emulate=True)
    out = mix[-m:]
    assert np.abs(out[:, 32:] - ref[:, 32:]).max() < 2e-3
    mu, mur = out[:, :32].reshape(m, 8, 4), ref[:, :32].reshape(m, 8, 4)
    assert np.quantile((mu[..., :3] * mur[..., :3]).sum(-1), 0.001) > 0.999
    np.testing.assert_allclose(mu[..., 3], mur[..., 3], rtol=2e-2)
