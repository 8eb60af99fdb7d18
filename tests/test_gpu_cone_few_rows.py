"""The cone forward projector for up to 32 detector rows (one per lane) and
just above, the source at any height among them, against the oracle, bit for
bit: single, batched, and with the SIRT residual.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reach", [0.5, 1.4])
@pytest.mark.parametrize("nv,above", [(2, 1), (3, 1), (4, 2), (16, 8), (17, 2), (24, 12), (31, 15),
                                      (32, 16), (32, 17), (32, 1), (33, 16), (40, 20)])
def test_forward_equals_the_oracle(nv, above, reach, cuda):
    """`above`: rows below the source."""
    import torch
    from ccpi.reconstruction.device import Plan
    g = O.cone_geometry((28, 24, 12), 1.0, 12, 33, 1.3, 50.0, 50.0, n_det_v=nv)
    g.v_pixels = (np.arange(nv) - above + 0.4) * (24.0 * reach / nv)
    p = Plan("cone", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape,
             source=g.source, detector_x=g.detector_x)
    rng = np.random.default_rng(nv)
    vol = rng.random((2,) + g.shape).astype(np.float32)
    t = torch.from_numpy(vol).to(cuda)
    ref = O.forward(g, vol[0])
    assert np.array_equal(p.forward(t[0].contiguous()).cpu().numpy(), ref)
    if ref.size % 4 == 0:
        both = p.forward_batch(t, torch.empty((2,) + p.sino_shape, device=cuda)).cpu().numpy()
        assert np.array_equal(both[0], ref)
        assert np.array_equal(both[1], O.forward(g, vol[1]))
    x = torch.zeros(p.shape, device=cuda)
    p.solve(O.SIRT, torch.from_numpy(ref).to(cuda), x, 2)
    assert np.array_equal(x.cpu().numpy(), O.solve(g, O.SIRT, ref, 2))
