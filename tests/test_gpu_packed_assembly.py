"""The element kernels that pack eight elements into a block, at the element counts of a
colour where a block is partly filled (1 to 9 elements), on distorted elements, against the
oracle's assembly (1e-12 relative, the tolerance of the element matrices)."""
import numpy as np
import pytest

import mastgpu as M
import oracle as O

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def distorted(nx, ny, nz):
    coords, conn = M.grid_hex8(nx, ny, nz)
    rng = np.random.default_rng(31)
    return coords + rng.uniform(-0.12, 0.12, coords.shape), conn, rng


def pattern(coords, conn):
    return O.csr_pattern(conn, coords.shape[0], 3)


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


# elements per colour: 1, 2, 3..4, 8, 9
@pytest.mark.parametrize("shape", [(2, 2, 2), (4, 2, 2), (7, 2, 2), (4, 4, 4), (6, 6, 2)])
def test_green_lagrange_tangent_and_residual(shape):
    coords, conn, rng = distorted(*shape)
    rho = rng.uniform(0.2, 1.0, conn.shape[0])
    X = rng.normal(scale=0.05, size=coords.shape[0] * 3)
    with M.Problem(M.PHYS_HEX8_NONLINEAR, coords, conn, M.SIMP_MATERIAL) as p:
        p.set_design(rho)
        R = p.residual_and_jacobian(X)
        vals = p.get_csr()[2]
        R_only = p.residual_and_jacobian(X, want_J=False)
    E, _ = O.simp_modulus(O.simp_desc(1, 1, 1), rho)
    rp, cols = pattern(coords, conn)
    ref, R_ref = O.assemble_hex8_gl(coords, conn, E, 0.3, X, None, rp, cols, None)
    assert rel(vals, ref) < RTOL and rel(R, R_ref) < RTOL
    assert np.array_equal(R, R_only)


@pytest.mark.parametrize("shape", [(2, 2, 2), (4, 2, 2), (7, 2, 2), (4, 4, 4), (6, 6, 2)])
def test_linear_stiffness(shape):
    coords, conn, rng = distorted(*shape)
    rho = rng.uniform(0.2, 1.0, conn.shape[0])
    with M.Problem(M.PHYS_HEX8, coords, conn, M.SIMP_MATERIAL) as p:
        p.set_design(rho)
        p.residual_and_jacobian(np.zeros(p.n_dofs), want_R=False)
        vals = p.get_csr()[2]
    E, _ = O.simp_modulus(O.simp_desc(1, 1, 1), rho)
    rp, cols = pattern(coords, conn)
    assert rel(vals, O.assemble_hex8(coords, conn, E, 0.3, rp, cols)) < RTOL


# 32 elements a block: 31, 32, 33, 64 and 65 elements
@pytest.mark.parametrize("nx", [31, 32, 33, 64, 65])
def test_element_energies(nx):
    """dC/drho_e = -dE_e u_e . K1_e u_e at an arbitrary u (zero on the fixed dofs)."""
    coords, conn, rng = distorted(nx, 1, 1)
    rho = rng.uniform(0.2, 1.0, nx)
    u = rng.normal(size=coords.shape[0] * 3)
    fixed = np.arange(12)
    with M.Problem(M.PHYS_HEX8, coords, conn, M.SIMP_MATERIAL, fixed_dofs=fixed) as p:
        p.set_design(rho)
        _, dc = p.compliance(X=u)
    _, dE = O.simp_modulus(O.simp_desc(1, 1, 1), rho)
    uf = u.copy()
    uf[fixed] = 0.0
    ref = []
    for e in range(nx):
        ue = uf.reshape(-1, 3)[conn[e]].T.reshape(-1)
        ref.append(-dE[e] * ue @ O.hex8_internal(coords[conn[e]], 1.0, 0.3)[1] @ ue)
    assert rel(dc, np.array(ref)) < RTOL
