"""The folded grid filter at the edges of its tiles (32 x 4 points, chunks of z planes), for
every ball of cells it has a kernel for, masked and transposed, against shifted sums in
numpy (the tolerance of the other filter tests)."""
import numpy as np
import pytest

import mastgpu as M

pytestmark = pytest.mark.gpu


def shifted(v, radius, h):
    """sum_o (r - |o h|) v at every cell, cells outside the grid as 0; v is (nz, ny, nx)"""
    n = [int(radius / s) for s in h]
    p = np.pad(v, [(n[2], n[2]), (n[1], n[1]), (n[0], n[0])])
    out = np.zeros_like(v)
    for c in range(-n[2], n[2] + 1):
        for b in range(-n[1], n[1] + 1):
            for a in range(-n[0], n[0] + 1):
                w = radius - np.sqrt((a * h[0]) ** 2 + (b * h[1]) ** 2 + (c * h[2]) ** 2)
                if w > 0:
                    out += w * p[n[2] + c:n[2] + c + v.shape[0], n[1] + b:n[1] + b + v.shape[1],
                                 n[0] + a:n[0] + a + v.shape[2]]
    return out


def check(nx, ny, nz, radius, h=(1.0, 1.0, 1.0)):
    rng = np.random.default_rng(41)
    shape = (max(nz, 1), ny, nx)
    hh = h if nz else (h[0], h[1], 1e30)
    x, g = rng.uniform(0.01, 1.0, shape), rng.normal(size=shape)
    for dv in (None, rng.random(shape) < 0.8):
        m = np.ones(shape, bool) if dv is None else dv
        S = shifted(np.ones(shape), radius, hh)
        fwd = np.where(m, shifted(x, radius, hh) / S, x)
        back = shifted(np.where(m, g / S, 0.0), radius, hh) + np.where(m, 0.0, g)
        with M.Filter.grid(nx, ny, nz, radius, dv=None if dv is None else dv.reshape(-1).astype(np.uint8), h=h) as f:
            assert np.abs(f.apply(x.reshape(-1)) - fwd.reshape(-1)).max() < 1e-13 * np.abs(fwd).max()
            assert np.abs(f.apply(g.reshape(-1), transpose=True) - back.reshape(-1)).max() < 1e-13 * np.abs(back).max()


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 6, 8, 9, 10, 11, 12, 13, 14, 16])
def test_every_ball(d):
    check(37, 9, 11, np.sqrt(d) + 0.01)


@pytest.mark.parametrize("dims", [(1, 1, 1), (31, 3, 2), (32, 4, 1), (33, 5, 7), (64, 8, 40), (65, 61, 0), (5, 130, 3)])
@pytest.mark.parametrize("radius", [1.5, 2.5, 3.5])
def test_tile_edges(dims, radius):
    check(*dims, radius)


def test_uneven_spacing_takes_the_general_form():
    check(19, 8, 6, 2.5, h=(1.0, 0.8, 1.3))
