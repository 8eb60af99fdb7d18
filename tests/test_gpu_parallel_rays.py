"""The parallel forward projector on either side of the ray counts where rays
begin to share warps, and with up to eight slices per lane, against the
oracle, bit for bit.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# slices, angles (of 101 detector columns)
CASES = [(4, 1), (4, 43), (4, 44), (16, 43), (16, 44), (20, 27), (20, 28), (32, 28),
         (36, 27), (36, 28), (64, 28), (129, 3), (131, 28), (255, 7), (257, 7), (263, 3)]


@pytest.mark.parametrize("nz,na", CASES)
def test_forward_equals_the_oracle(nz, na, cuda):
    import torch
    from ccpi.reconstruction.device import Plan
    rng = np.random.default_rng(nz * 100 + na)
    shape = (int(rng.integers(30, 80)), int(rng.integers(30, 80)), nz)
    g = O.parallel_geometry(shape, na, 101, cor_shift=0.37, span=2 * np.pi)
    p = Plan("parallel", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape)
    vol = rng.random(g.shape).astype(np.float32)
    out = p.forward(torch.from_numpy(vol).to(cuda)).cpu().numpy()
    assert np.array_equal(out, O.forward(g, vol))
    x = torch.full(g.shape, 0.5, device=cuda)
    p.solve(1, torch.from_numpy(out).to(cuda), x, 2)
    ref = O.solve(g, O.SIRT, out, 2, x0=np.full(g.shape, 0.5, np.float32))
    assert np.array_equal(x.cpu().numpy(), ref)
