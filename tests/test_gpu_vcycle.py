"""The multigrid V-cycle's forms and the device loop around it: smoothers of several degrees,
chains that start at the design's own grid (at most 5,000 nodes) or below it, grids at the edges
of the level operator's tiles (31 x 15 owned nodes), and solves longer than one loop launch."""
import functools

import numpy as np
import pytest

import mastgpu as M
import oracle as O

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def reference(shape):
    nx, ny, nz = shape
    rho = np.random.default_rng(31).uniform(0.01, 1.0, nx * ny * nz)
    _, dc, r = O.simp_solve(O.simp_desc(nx, ny, nz, rtol=1e-12, maxit=10 ** 6), rho)
    return rho, r.compliance, dc


# 4 x 4 x 4: the smallest chain of two levels; 16^3 (4,913 nodes): the largest cube solved from its
# own grid; 17 x 16 x 16 (5,202 nodes): level by level; 30/31/32 x 14/15/16: one node short of a tile,
# a whole one, one node over; 2 x 1 x 26: the second level (56 nodes) leaves two of sixteen CTAs
# without nodes, the third (32) none
SHAPES = [(4, 4, 4), (9, 8, 3), (16, 16, 16), (17, 16, 16), (30, 14, 9), (31, 15, 10), (32, 16, 9), (2, 1, 26)]


@pytest.mark.parametrize("degree", [1, 2, 3, 5])
@pytest.mark.parametrize("shape", SHAPES)
def test_smoother_degrees_match_the_oracle(shape, degree):
    """A preconditioner changes the path, not the result: residual 1e-8, results 1e-6, as for the
    other mixed solves.  A smoother that is not symmetric or not positive breaks the solve down."""
    nx, ny, nz = shape
    rho, c_ref, dc_ref = reference(shape)
    o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-8, inner_rtol=1e-2, timeout_s=300.0)
    o.smooth_degree = degree
    with M.simp_cantilever(nx, ny, nz) as p:
        p.set_design(rho)
        _, rep = p.solve(o)
        c, dc = p.compliance()
    with M.Batch([dict(nx=nx, ny=ny, nz=nz, rho=rho, spans=[(0, ny)]), dict(nx=6, ny=5, nz=4, rho=np.resize(rho, 120), spans=[(0, 5)])]) as b:
        _, reps = b.solve(o)
        cb, dcb, _ = b.results(0)
    # both forms apply the same preconditioner up to rounding
    assert abs(rep.krylov_iterations - reps[0].krylov_iterations) <= 2, (rep.krylov_iterations, reps[0].krylov_iterations)
    for st, relres, ci, di in ((rep.status, rep.relres, c, dc), (reps[0].status, reps[0].relres, cb[0], dcb[0])):
        assert st == 0 and relres <= 1e-8, (st, relres)
        assert abs(ci - c_ref) / c_ref < 1e-6
        assert np.abs(di - dc_ref).max() / np.abs(dc_ref).max() < 1e-6


def test_thin_batched_chains_on_few_ctas(monkeypatch):
    """Chains of 1,024 nodes with one, two and sixteen CTAs: the same bits.  Beside them a design too
    slender for FP32 (its solve breaks down), whose 1,024 nodes with all coarser levels do not fit one
    CTA: its chain starts a level lower and the others keep theirs."""
    shapes = [(63, 3, 3), (40, 4, 4), (255, 1, 1)]
    o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-8, inner_rtol=1e-2, timeout_s=300.0)
    out = []
    for cap in ("1", "2", "16"):
        monkeypatch.setenv("MASTGPU_BOTTOM_CLUSTER", cap)
        with M.Batch([dict(nx=s[0], ny=s[1], nz=s[2], rho=reference(s)[0] if s[2] > 1 else np.ones(255), spans=[(0, s[1])])
                      for s in shapes]) as b:
            _, reps = b.solve(o, raise_on_error=False)
            out.append([b.results(d)[:2] for d in (0, 1)])
        for s, rep, (c, dc) in zip(shapes, reps, out[-1]):
            _, c_ref, dc_ref = reference(s)
            assert rep.status == 0 and rep.relres <= 1e-8
            assert abs(c[0] - c_ref) / c_ref < 1e-6
            assert np.abs(dc[0] - dc_ref).max() / np.abs(dc_ref).max() < 1e-6
    for o2 in out[1:]:
        for (c, dc), (c0, dc0) in zip(o2, out[0]):
            assert np.array_equal(c, c0) and np.array_equal(dc, dc0)


def test_solve_longer_than_one_loop_launch():
    """Jacobi-preconditioned solves of some hundred iterations, two per loop body and 64 bodies a
    launch: the same iterations and the same bits as with 16 per body (one launch or two)."""
    nx, ny, nz = 40, 4, 4
    rho, c_ref, _ = reference((nx, ny, nz))
    out = []
    for chunk in (2, 16):
        o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-8, inner_rtol=1e-3, timeout_s=300.0)
        o.preconditioner, o.graph_chunk = M.PC_JACOBI, chunk
        with M.simp_cantilever(nx, ny, nz) as p:
            p.set_design(rho)
            u, rep = p.solve(o)
            c, _ = p.compliance()
        assert rep.status == 0 and rep.krylov_iterations > 2 * 64 * 2
        assert abs(c - c_ref) / c_ref < 1e-6
        out.append((u, rep.krylov_iterations, rep.refinements))
    assert out[0][1:] == out[1][1:] and np.array_equal(out[0][0], out[1][0])


def test_iteration_cap_ends_the_loop():
    """Caps that are reached: every inner solve stops after one iteration and the third refinement is
    the last; the status says that the solve did not converge."""
    rho, _, _ = reference((9, 8, 3))
    o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-12, inner_rtol=1e-6, timeout_s=300.0)
    o.max_iterations, o.max_refinements = 1, 3
    with M.simp_cantilever(9, 8, 3) as p:
        p.set_design(rho)
        rc, rep = p.solve_resident(o)
    assert rc == rep.status != 0
    assert rep.refinements == 3 and rep.krylov_iterations == 3
