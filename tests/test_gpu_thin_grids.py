"""Structured grids one element thick: half or more of the structured colours have no element.
Assembly against the oracle's (1e-12 relative, the tolerance of the element matrices), on
distorted elements, and a solve through the grid's own entry point."""
import numpy as np
import pytest

import mastgpu as M
import oracle as O

pytestmark = pytest.mark.gpu

RTOL = 1e-12
SHAPES = [(1, 1, 1), (5, 4, 1), (1, 3, 5), (4, 1, 3), (2, 1, 1)]


def distorted(shape):
    coords, conn = M.grid_hex8(*shape)
    rng = np.random.default_rng(5)
    return coords + rng.uniform(-0.12, 0.12, coords.shape), conn, rng


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("shape", SHAPES)
def test_linear_assembly(shape):
    coords, conn, rng = distorted(shape)
    rho = rng.uniform(0.2, 1.0, conn.shape[0])
    with M.Problem(M.PHYS_HEX8, coords, conn, M.SIMP_MATERIAL, grid=shape) as p:
        p.set_design(rho)
        p.residual_and_jacobian(np.zeros(p.n_dofs), want_R=False)
        vals = p.get_csr()[2]
    E, _ = O.simp_modulus(O.simp_desc(1, 1, 1), rho)
    rp, cols = O.csr_pattern(conn, coords.shape[0], 3)
    assert rel(vals, O.assemble_hex8(coords, conn, E, 0.3, rp, cols)) < RTOL


@pytest.mark.parametrize("shape", SHAPES)
def test_green_lagrange_assembly(shape):
    coords, conn, rng = distorted(shape)
    rho = rng.uniform(0.2, 1.0, conn.shape[0])
    X = rng.normal(scale=0.05, size=coords.shape[0] * 3)
    with M.Problem(M.PHYS_HEX8_NONLINEAR, coords, conn, M.SIMP_MATERIAL, grid=shape) as p:
        p.set_design(rho)
        R = p.residual_and_jacobian(X)
        vals = p.get_csr()[2]
    E, _ = O.simp_modulus(O.simp_desc(1, 1, 1), rho)
    rp, cols = O.csr_pattern(conn, coords.shape[0], 3)
    ref, R_ref = O.assemble_hex8_gl(coords, conn, E, 0.3, X, None, rp, cols, None)
    assert rel(vals, ref) < RTOL and rel(R, R_ref) < RTOL


def test_plain_solve():
    nx, ny, nz = 6, 4, 1
    rho = np.random.default_rng(6).uniform(0.2, 1.0, nx * ny * nz)
    u_ref, dc_ref, r = O.simp_solve(O.simp_desc(nx, ny, nz, rtol=1e-13), rho)
    with M.simp_cantilever(nx, ny, nz) as p:
        p.set_design(rho)
        u, rep = p.solve(M.default_opts(rtol=1e-12))
        c, dc = p.compliance()
    assert rep.status == 0
    assert rel(u, u_ref) < 1e-9 and abs(c - r.compliance) / r.compliance < 1e-10 and rel(dc, dc_ref) < 1e-9


def test_heat_strip():
    """A strip one element high: two of the four colours of a 2D grid are empty."""
    nx = 7
    coords, conn = M.grid_quad4(nx, 1, 1.0, 0.2)
    X = np.random.default_rng(7).uniform(0.0, 1.0, coords.shape[0])
    mat = dict(M.SIMP_MATERIAL, k0=1.3, k_beta=0.05)
    with M.Problem(M.PHYS_HEAT, coords, conn, mat, grid=(nx, 1, 0)) as p, M.Problem(M.PHYS_HEAT, coords, conn, mat) as q:
        R, Rq = p.residual_and_jacobian(X), q.residual_and_jacobian(X)
        vals, vq = p.get_csr()[2], q.get_csr()[2]
    # the greedy colouring of a general mesh adds the elements of a node in another order
    assert rel(R, Rq) < RTOL and rel(vals, vq) < RTOL
