"""The scatter's form for detectors that reach past the volume's ends, at each
number of rows per lane, and on either side of the rule between its forms:
within the projector tolerance of the oracle; CGLS with it (on a sinogram
already scaled) as close to FP64 as the float oracle.
"""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2

pytestmark = pytest.mark.gpu

ROWS = [6, 30, 32, 34, 64, 96, 100, 128, 190, 200, 288, 300]


@pytest.mark.parametrize("reach", [0.75, 0.9, 1.3, 2.5])
@pytest.mark.parametrize("nv", ROWS)
def test_scatter_past_the_ends(nv, reach, cuda):
    import torch
    from ccpi.reconstruction.device import Plan
    g = O.cone_geometry((26, 21, 30), 1.0, 11, 37, 1.1, 60.0, 60.0, n_det_v=nv)
    # the outermost rows' height on the axis over the volume's half height;
    # the source above or below the middle
    g.v_pixels = (np.arange(nv) - (nv - 1) / 2.0) * (60.0 * reach / nv) + (0.1 if nv % 3 else 3.2)
    p = Plan("cone", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape,
             source=g.source, detector_x=g.detector_x)
    rng = np.random.default_rng(nv)
    pix = rng.random(g.sino_shape).astype(np.float32)
    t = torch.from_numpy(pix).to(cuda)
    p.set_cone_backprojector(1)
    ref = O.backward(g, pix)
    assert np.abs(p.backward(t).cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()
    x = torch.zeros(p.shape, device=cuda)
    p.solve(O.CGLS, t, x, 2)
    want = O.solve(g, O.CGLS, pix.astype(np.float64), 2, fp64=True)
    bound = max(1e-4, 2.0 * rel_l2(O.solve(g, O.CGLS, pix, 2), want))
    assert rel_l2(x.cpu().numpy(), want) <= bound
