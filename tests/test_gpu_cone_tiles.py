"""The tiled cone back projector against the oracle, bit for bit, where its
tiles, slice chunks, staged patches and row loops end.  Every volume but the
last is large enough (more than 2^19 voxels, or taller than 256) for tiles.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

CASES = {
    # ragged tiles and a last chunk of two slices
    "ragged": dict(shape=(97, 83, 66), na=7, nd=70, nv=62, pix=2.0, s=150.0),
    # several slices from one row to the next
    "coarse rows": dict(shape=(150, 120, 31), na=6, nd=60, nv=14, pix=6.0, s=260.0),
    # many rows per slice next to the source: patches taken in parts
    "near source": dict(shape=(88, 88, 70), na=9, nd=300, nv=260, pix=0.7, s=75.0),
    # one part still too large to stage: the sinogram itself
    "fine detector": dict(shape=(72, 72, 104), na=3, nd=440, nv=560, pix=0.4, s=90.0),
    # rows that leave through the far end of the column
    "edge rows": dict(shape=(90, 90, 66), na=8, nd=110, nv=150, pix=1.0, s=120.0),
    # a row at the source height (NaN as in the oracle), odd everything
    "odd": dict(shape=(85, 87, 73), na=5, nd=91, nv=75, pix=1.5, s=130.0),
    "tall": dict(shape=(5, 9, 300), na=11, nd=17, nv=330, pix=0.9, s=50.0),
    "small": dict(shape=(30, 22, 40), na=13, nd=31, nv=36, pix=1.2, s=50.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tiles_equal_the_oracle(name, cuda):
    import torch
    from ccpi.reconstruction.device import Plan
    c = CASES[name]
    g = O.cone_geometry(c["shape"], 1.0, c["na"], c["nd"], c["pix"], c["s"], c["s"],
                        n_det_v=c["nv"])
    p = Plan("cone", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape,
             source=g.source, detector_x=g.detector_x)
    rng = np.random.default_rng(sum(map(ord, name)))
    pix = rng.random((2,) + tuple(g.sino_shape)).astype(np.float32)
    ref = O.backward(g, pix[0])
    t = torch.from_numpy(pix).to(cuda)
    one = p.backward(t[0].contiguous()).cpu().numpy()
    assert np.array_equal(one, ref, equal_nan=True)
    if ref.size % 4 == 0 and pix[0].size % 4 == 0:
        both = p.backward_batch(t, torch.empty((2,) + p.shape, device=cuda)).cpu().numpy()
        assert np.array_equal(both[0], ref, equal_nan=True)
        assert np.array_equal(both[1], O.backward(g, pix[1]), equal_nan=True)


@pytest.mark.parametrize("nv", [6, 24, 32, 40, 64, 96, 100, 128, 160, 192, 200, 256, 288, 300])
def test_scatter_at_every_row_count(nv, cuda):
    """The scatter's passes of rows (1 to 8 per lane, split by the source or
    not): within the projector tolerance of the oracle."""
    import torch
    from ccpi.reconstruction.device import Plan
    g = O.cone_geometry((26, 21, 30), 1.0, 11, 37, 1.1, 60.0, 60.0, n_det_v=nv)
    # rows over the same height, the source above or below the middle
    g.v_pixels = (np.arange(nv) - (nv - 1) / 2.0) * (34.0 / nv) + (0.1 if nv % 3 else 3.2)
    p = Plan("cone", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape,
             source=g.source, detector_x=g.detector_x)
    rng = np.random.default_rng(nv)
    pix = rng.random(g.sino_shape).astype(np.float32)
    ref = O.backward(g, pix)
    p.set_cone_backprojector(1)
    out = p.backward(torch.from_numpy(pix).to(cuda)).cpu().numpy()
    assert np.abs(out - ref).max() <= 1e-5 * np.abs(ref).max()
    vol = rng.random(g.shape).astype(np.float32)
    assert np.array_equal(p.forward(torch.from_numpy(vol).to(cuda)).cpu().numpy(),
                          O.forward(g, vol))
