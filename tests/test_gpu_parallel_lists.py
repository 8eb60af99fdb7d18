"""The parallel forward projector where a ray lists many 32 x 32 blocks,
against the oracle, bit for bit: rays almost parallel to an axis on a block
boundary (two blocks of every block column), diagonals through block corners
(three), and grids whose lists are longer than the staging area.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

F32_TURN = float(np.float32(2 * np.pi))   # |sin| just above the parallel rule's limit
F32_DIAGONAL = float(np.float32(np.pi / 4))

CASES = {
    "two blocks a column": ((2048, 64, 4), F32_TURN, 9, 0.0),
    "below the boundary": ((2048, 64, 4), F32_TURN, 9, -5e-4),
    "along y": ((64, 2048, 4), float(np.float32(np.pi / 2)), 9, 0.0),
    "diagonal": ((2048, 2048, 1), F32_DIAGONAL, 5, 0.0),
    "odd slices": ((1024, 64, 5), F32_TURN, 9, -5e-4),
    "one ray per warp": ((4800, 64, 68), F32_TURN, 5, -5e-4),
    "wide": ((34000, 32, 4), 0.003, 9, 0.0),
    "wider than any list": ((300000, 40, 1), 1e-4, 5, 0.0),
    "wider than 2^20": ((1100000, 3, 1), 2e-6, 5, 0.0),
    "tall": ((40, 300000, 1), float(np.pi / 2 - 1e-4), 5, 0.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_long_block_lists_equal_the_oracle(name, cuda):
    import torch
    from ccpi.reconstruction.device import Plan
    shape, angle, nh, shift = CASES[name]
    g = O.parallel_geometry(shape, 3, nh, nv=max(shape[2], 1))
    g.angles = np.array([angle, 0.0, angle + 0.7])
    g.h_pixels = np.arange(nh) - (nh - 1) / 2.0 + shift
    p = Plan("parallel", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape)
    rng = np.random.default_rng(nh)
    vol = rng.random(g.shape, dtype=np.float32)
    out = p.forward(torch.from_numpy(vol).to(cuda)).cpu().numpy()
    assert np.array_equal(out, O.forward(g, vol))
