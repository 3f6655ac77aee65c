"""Single plate-like designs: the tables of a bottom chain grow with NX NY of its levels, so the
first level that is small enough in nodes may be too wide for the clusters.  Its chain then starts
a level lower (and the coarsest grid is still solved directly) instead of nowhere."""
import numpy as np
import pytest

import mastgpu as M
import oracle as O

pytestmark = pytest.mark.gpu


# the widest levels of at most 5,000 nodes: the designs' own grids (35 x 35 x 4 and 37 x 35 x 3
# nodes), the second level (34 x 34 x 4, 41 x 33 x 3 nodes)
@pytest.mark.parametrize("shape", [(34, 34, 3), (36, 34, 2), (66, 66, 6), (80, 64, 4)])
def test_flat_design_keeps_a_chain(shape):
    nx, ny, nz = shape
    rho = np.random.default_rng(17).uniform(0.2, 1.0, nx * ny * nz)
    _, dc_ref, r = O.simp_solve(O.simp_desc(nx, ny, nz, rtol=1e-12, maxit=10 ** 6), rho)
    o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-8, inner_rtol=1e-3, timeout_s=300.0)
    with M.simp_cantilever(nx, ny, nz) as p:
        p.set_design(rho)
        p.solve_resident(o)  # tables
        n0 = M.lib().mg_launch_count()
        rc, rep = p.solve_resident(o)
        launches = M.lib().mg_launch_count() - n0
        c, dc = p.compliance()
    assert rc == rep.status == 0 and rep.relres <= 1e-8
    assert abs(c - r.compliance) / r.compliance < 1e-6
    assert np.abs(dc - dc_ref).max() / np.abs(dc_ref).max() < 1e-6
    # A CG iteration: six launches for each level above the chain (two at the most here), the chain,
    # r.z, the operator, the update, half a loop gate: 16.5.  Without a chain it is 31 or more (five
    # levels, a coarsest smoother of degree eight).  Steps come in pairs: one more a refinement.
    its = rep.krylov_iterations + rep.refinements + 1
    assert launches <= 17 * its + 12 * (rep.refinements + 1) + 20, (launches, rep.krylov_iterations, rep.refinements)
