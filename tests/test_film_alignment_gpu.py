"""The film's paired sums: a film that does not start on a 16-byte boundary gets the same sums, with every
reconstruction filter's weights."""
import numpy as np
import pytest

import oracle
from liar_b200 import cameras, render as R, scenery, shaders, spectra, textures, tracers
from liar_b200.kernel import default_context

pytestmark = pytest.mark.gpu

def panel(spectrum):
    wall = scenery.Parallelogram((-5, -5, 0), (10, 0, 0), (0, 10, 0))
    wall.shader = shaders.Unshaded(textures.Constant(spectrum))
    cam = cameras.PerspectiveCamera()
    cam.position = (0, 0, 4)
    cam.sky = (0, 1, 0)  # (before looking along the default sky's axis)
    cam.lookAt((0, 0, 0))
    cam.aspectRatio = 1
    return scenery.List([wall]), cam


@pytest.mark.parametrize("filter_, param", [(0, 0.0), (1, 1.5), (2, 0.0)])
@pytest.mark.parametrize("offset", [0, 1, 4, 7])
def test_film_of_any_alignment(filter_, param, offset):
    import torch
    scene, cam = panel(spectra.BlackBody(4000.0, 1.0))
    flat = R.flatten(scene)
    desc = R.render_desc(cam, 33, 21, 4, tracers.AdjointPhotonTracer(), seed=1, filter=filter_, filter_param=param)
    gs = R.GpuScene(default_context(), flat)
    buf = torch.zeros(33 * 21 * 8 + 64, device="cuda")
    torch.cuda.synchronize()
    gs.render_device(desc, buf[offset:].data_ptr())
    gs.ctx.synchronize()
    got = buf.cpu().numpy()
    assert np.all(got[:offset] == 0) and np.all(got[offset + 33 * 21 * 8:] == 0)
    c = oracle.RenderScene(flat).render(desc)
    # up to 25 pixels' samples of 4 each, with weights of either sign, relative to the largest sum
    np.testing.assert_allclose(got[offset:offset + 33 * 21 * 8].reshape(21, 33, 8), c, rtol=0,
                               atol=float(np.abs(c).max()) * 400 * 2.0 ** -24)
