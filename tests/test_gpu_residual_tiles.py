"""The FP64 residual of the mixed solves on grids around its tile edges (16 x 8 owned nodes, the last
tile of a side one more; 12 node planes at most)."""
import numpy as np
import pytest

import mastgpu as M
import oracle as O

pytestmark = pytest.mark.gpu


# one element short of a tile, a whole one, one over, in x and y; several tiles; depths of one plane
# (single designs), of twelve and a remainder (batches)
@pytest.mark.parametrize("shape", [(15, 7, 5), (16, 8, 11), (17, 9, 12), (33, 15, 3), (32, 17, 13), (2, 1, 26)])
def test_residual_tiles_match_the_oracle(shape):
    """A residual that misses a node's element converges to the wrong solution or not at all.  Cold and
    warm starts (the first residual of a cold start is the load).  Mixed-form tolerances (1e-8
    residual, 1e-6 results)."""
    nx, ny, nz = shape
    rho = np.random.default_rng(41).uniform(0.01, 1.0, nx * ny * nz)
    o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-8, inner_rtol=1e-2, timeout_s=300.0)
    with M.simp_cantilever(nx, ny, nz) as p:
        p.set_design(rho)
        u0, rep = p.solve(o)
        c, dc = p.compliance()
        o.warm_start = 1
        u1, rep1 = p.solve(o, X=u0)
    o.warm_start = 0
    with M.Batch([dict(nx=nx, ny=ny, nz=nz, rho=rho, spans=[(0, ny)])]) as b:
        _, reps = b.solve(o)
        cb, dcb, _ = b.results(0)
    # the solution that was accepted is accepted again, unchanged
    assert rep1.status == 0 and rep1.krylov_iterations == 0 and np.array_equal(u0, u1)
    assert rep1.relres == rep.relres
    _, dc_ref, r = O.simp_solve(O.simp_desc(nx, ny, nz, rtol=1e-12, maxit=10 ** 6), rho)
    for st, relres, ci, di in ((rep.status, rep.relres, c, dc), (reps[0].status, reps[0].relres, cb[0], dcb[0])):
        assert st == 0 and relres <= 1e-8, (st, relres)
        assert abs(ci - r.compliance) / r.compliance < 1e-6
        assert np.abs(di - dc_ref).max() / np.abs(dc_ref).max() < 1e-6
