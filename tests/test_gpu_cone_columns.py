"""The tiled cone back projector with detector columns that are not exactly
evenly spaced, against the oracle, bit for bit: positions rounded to float32
(as read from a file), jittered, widening, and far off the axis.  The rays of
a voxel column are the reference's (c2D.cpp:831-895), whose range of columns
comes from the first two positions alone.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def f32(n, pitch):
    return ((np.arange(n) - (n - 1) / 2.0) * pitch).astype(np.float32).astype(np.float64)


def jittered(n, pitch, by):
    rng = np.random.default_rng(n)
    return (np.arange(n) - (n - 1) / 2.0 + rng.uniform(-by, by, n)) * pitch


def widening(n, pitch):
    i = np.arange(n, dtype=np.float64)
    h = pitch * (i + 4e-4 * i * i)
    return h - h.mean()


COLUMNS = {
    "float32, 2048 of 0.15": lambda: f32(2048, 0.15),
    "float32, 1024 of 0.3": lambda: f32(1024, 0.3),
    "jitter 3 %": lambda: jittered(220, 1.5, 0.03),
    "jitter 0.5 %": lambda: jittered(220, 1.5, 0.005),
    "widening": lambda: widening(200, 1.5),
    "even": lambda: (np.arange(512) - 255.5) * 0.6,
    "off the axis": lambda: (np.arange(24) + 400.0) * 0.3,
}


@pytest.mark.parametrize("name", sorted(COLUMNS))
def test_uneven_columns_equal_the_oracle(name, cuda):
    import torch
    from ccpi.reconstruction.device import Plan
    h = COLUMNS[name]()
    # far enough that no voxel column sees more than 24 rays of an angle, the
    # back projector's limit
    s = 700.0 if len(h) > 1024 else 220.0
    g = O.cone_geometry((136, 128, 31), 1.0, 7, len(h), 1.0, s, s, n_det_v=8)
    g.angles = g.angles + 0.1
    g.h_pixels = h
    g.v_pixels = (np.arange(8) - 3.5) * 8.0
    p = Plan("cone", g.angles, g.h_pixels, g.v_pixels, g.origin, g.size, g.shape,
             source=g.source, detector_x=g.detector_x)
    rng = np.random.default_rng(len(h))
    pix = rng.random(g.sino_shape).astype(np.float32)
    out = p.backward(torch.from_numpy(pix).to(cuda)).cpu().numpy()
    assert np.array_equal(out, O.backward(g, pix), equal_nan=True)
