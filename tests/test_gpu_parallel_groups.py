"""The parallel forward projector for few slices, odd slices and any map of
rows to slices, against the oracle, bit for bit: at the slice counts where
the lanes per ray, the slices per lane and the launches change.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# nz, detector rows, row pitch in slices, first row's height over the
# volume's lower face
MAPS = [(4, 4, 1.0, 0.5), (16, 16, 1.0, 0.5), (20, 20, 1.0, 0.5), (32, 32, 1.0, 0.5),
        (36, 36, 1.0, 0.5), (64, 64, 1.0, 0.5), (68, 66, 1.0, 0.5),
        (1, 1, 1.0, 0.5), (15, 15, 1.0, 0.5), (17, 17, 1.0, 0.5), (33, 33, 1.0, 0.5),
        (65, 65, 1.0, 0.5), (131, 131, 1.0, 0.5),
        (12, 24, 0.5, 0.25), (132, 264, 0.5, 0.25), (9, 36, 0.25, 0.125),
        (264, 264, 1.0, 0.5), (20, 13, 1.3, 0.2), (18, 40, 0.7, -4.0)]


@pytest.mark.parametrize("nz,nv,pitch,first", MAPS)
def test_forward_equals_the_oracle(nz, nv, pitch, first, cuda):
    import torch
    from ccpi.reconstruction.device import Plan
    rng = np.random.default_rng(nz * 1000 + nv)
    shape = (int(rng.integers(20, 75)), int(rng.integers(20, 75)), nz)
    # a number of angles that leaves the last warp's rays partly idle, the
    # axis-parallel directions among them
    g = O.parallel_geometry(shape, 21, 90, nv=max(nv, 2), cor_shift=0.37, span=2 * np.pi)
    g.v_pixels = g.origin[2] + first + pitch * np.arange(nv)
    p = Plan("parallel", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape)
    vol = rng.random(g.shape).astype(np.float32)
    out = p.forward(torch.from_numpy(vol).to(cuda)).cpu().numpy()
    assert np.array_equal(out, O.forward(g, vol))


@pytest.mark.parametrize("nz", [4, 24, 33])
def test_rays_of_a_warp_of_very_different_lengths(nz, cuda):
    """A wide grid under a wider detector and few angles: some rays of a warp
    cross hundreds of cells while others miss the volume."""
    import torch
    from ccpi.reconstruction.device import Plan
    rng = np.random.default_rng(nz)
    g = O.parallel_geometry((420, 380, nz), 13, 560, cor_shift=0.37, span=2 * np.pi)
    p = Plan("parallel", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape)
    vol = rng.random(g.shape).astype(np.float32)
    out = p.forward(torch.from_numpy(vol).to(cuda)).cpu().numpy()
    assert np.array_equal(out, O.forward(g, vol))
