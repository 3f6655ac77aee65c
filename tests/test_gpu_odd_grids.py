"""Multigrid on grids with odd sides: an odd side is padded by one void element when it is
coarsened, so every design reaches a directly solved coarsest grid."""
import numpy as np
import pytest

import mastgpu as M
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 3, 3), (7, 3, 3), (9, 5, 4), (23, 13, 9), (33, 15, 17), (31, 17, 2), (40, 4, 4), (30, 5, 1)])
def test_odd_grid_design_matches_the_oracle(shape):
    """Smallest grid with a coarse level, odd in one to three sides at one or more levels,
    and sides of one and two elements.  Mixed-form tolerances (1e-8 residual, 1e-6 results)."""
    nx, ny, nz = shape
    rho = np.random.default_rng(21).uniform(0.01, 1.0, nx * ny * nz)
    o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-8, inner_rtol=1e-2, timeout_s=300.0)
    with M.simp_cantilever(nx, ny, nz) as p:
        p.set_design(rho)
        _, rep = p.solve(o)
        c, dc = p.compliance()
    with M.Batch([dict(nx=nx, ny=ny, nz=nz, rho=rho, spans=[(0, ny)])]) as b:
        rc, reps = b.solve(o)
        cb, dcb, _ = b.results(0)
    _, dc_ref, r = O.simp_solve(O.simp_desc(nx, ny, nz, rtol=1e-12, maxit=10 ** 6), rho)
    for st, relres, ci, di in ((rep.status, rep.relres, c, dc), (reps[0].status, reps[0].relres, cb[0], dcb[0])):
        assert st == 0 and relres <= 1e-8, (st, relres)
        assert abs(ci - r.compliance) / r.compliance < 1e-6
        assert np.abs(di - dc_ref).max() / np.abs(dc_ref).max() < 1e-6


@pytest.mark.parametrize("shape", [(23, 13, 9), (9, 7, 5)])
def test_clamped_far_face_of_an_odd_grid(shape):
    """Both x faces clamped on an odd length: the coarse nodes beyond the grid are
    constrained with the face.  Against the plain FP64 form of the same problem."""
    nx, ny, nz = shape
    NX, NY, NZ = nx + 1, ny + 1, nz + 1
    coords, conn = M.grid_hex8(nx, ny, nz)
    faces = np.concatenate([NX * np.arange(NY * NZ), nx + NX * np.arange(NY * NZ)])
    fixed = (faces[:, None] * 3 + np.arange(3)).reshape(-1)
    load = 3 * (nx // 2 + NX * (np.arange(NY) + NY * (NZ - 1))) + 2
    rho = np.random.default_rng(22).uniform(0.01, 1.0, nx * ny * nz)
    out = []
    with M.Problem(M.PHYS_HEX8, coords, conn, M.SIMP_MATERIAL, fixed_dofs=fixed, load_dofs=load,
                   load_values=np.full(NY, -1.0 / NY), grid=(nx, ny, nz)) as p:
        p.set_design(rho)
        for o in (M.default_opts(rtol=1e-12), M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-8, inner_rtol=1e-2)):
            _, rep = p.solve(o)
            assert rep.status == 0
            out.append(p.compliance())
    (c0, dc0), (c1, dc1) = out
    assert abs(c1 - c0) / abs(c0) < 1e-6
    assert np.abs(dc1 - dc0).max() / np.abs(dc0).max() < 1e-6
