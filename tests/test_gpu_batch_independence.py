"""A design's results do not depend on the batch around it, at sizes where a split of the work by
the whole batch would show: alone each of these designs is a small part of a wave of blocks, in
this batch (1.8 M dofs, 45 problems a level) every share of the GPU is small."""
import numpy as np
import pytest

import mastgpu as M

pytestmark = pytest.mark.gpu


def design(shape, seed):
    nx, ny, nz = shape
    rho = np.random.default_rng(seed).uniform(0.01, 1.0, nx * ny * nz)
    return dict(nx=nx, ny=ny, nz=nz, rho=rho, spans=[(0, ny)])


@pytest.mark.parametrize("smoother", [M.SMOOTHER_FACTORED, M.SMOOTHER_TENSOR])
def test_large_batch_and_alone_give_the_same_bits(smoother):
    small = [design(s, i) for i, s in enumerate([(16, 8, 8), (24, 12, 12), (48, 24, 24), (33, 15, 17)])]
    rest = [design((128, 64, 64), 10)] + [design((4, 4, 4), 11 + i) for i in range(40)]
    o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-8, inner_rtol=1e-3, timeout_s=300.0)
    o.smoother_operator = smoother
    with M.Batch(small + rest) as b:
        _, reps = b.solve(o)
        together = [b.results(d, want_u=True) for d in range(len(small))]
    for d, des in enumerate(small):
        with M.Batch([des]) as b:
            _, rep = b.solve(o)
            alone = b.results(0, want_u=True)
        assert rep[0].krylov_iterations == reps[d].krylov_iterations
        for a, t in zip(alone, together[d]):
            assert np.array_equal(a, t), d
