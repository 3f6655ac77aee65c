"""The one-kernel Krylov form (vectors resident in shared memory) at the sizes where its
shape changes: rows in registers or streamed, 1 to 3 dofs per node, rows longer than the
structured stencils, and the first size past it.  The reference is the residual of the
returned solution formed by numpy from the assembled CSR."""
import numpy as np
import pytest
import scipy.sparse as sp

import mastgpu as M

pytestmark = pytest.mark.gpu


def csr(p):
    rp, cols, vals = p.get_csr()
    return sp.csr_matrix((vals, cols, rp), shape=(p.n_dofs, p.n_dofs))


def check(p, o, times=2):
    """||F - K u|| <= rtol ||F|| up to the rounding of a recurrence residual; the same bits
    every time."""
    us = [p.solve(o)[0] for _ in range(times)]
    F = -p.residual_and_jacobian(np.zeros(p.n_dofs))
    assert np.linalg.norm(F - csr(p) @ us[0]) <= 2 * o.rtol * np.linalg.norm(F)
    for u in us[1:]:
        assert np.array_equal(u, us[0])


# nodes: 27 (fewer than SMs), 9,576 (the last with rows in registers on 152 SMs), 10,143
# (streamed), 226,981 (past the shared-memory form)
@pytest.mark.parametrize("shape", [(2, 2, 2), (37, 17, 13), (22, 20, 20), (60, 60, 60)])
def test_hex8(shape):
    rho = np.random.default_rng(5).uniform(0.3, 1.0, int(np.prod(shape)))
    with M.simp_cantilever(*shape) as p:
        p.set_design(rho)
        check(p, M.default_opts(rtol=1e-9))


def test_more_iterations_than_one_launch():
    """1,000-odd iterations: the state passes from launch to launch; an iteration cap is met exactly."""
    with M.simp_cantilever(60, 6, 6) as p:
        p.set_design(np.random.default_rng(6).uniform(0.05, 1.0, 60 * 36))
        check(p, M.default_opts(rtol=1e-9))
        for cap in (1, 255, 256, 257):
            _, rep = p.solve(M.default_opts(rtol=1e-9, max_iterations=cap), raise_on_error=False)
            assert (rep.status, rep.krylov_iterations) == (M.MG_ENOCONV, cap)


@pytest.mark.parametrize("n", [9, 140])
def test_membrane_two_dofs_per_node(n):
    coords, conn = M.grid_quad4(n, n)
    left = (n + 1) * np.arange(n + 1)
    mat = dict(E0=1.0, Emin=1e-9, nu=0.3, penal=3.0, thickness=0.1, k0=0.0, k_beta=0.0)
    with M.Problem(M.PHYS_MEMBRANE, coords, conn, mat, fixed_dofs=np.concatenate([2 * left, 2 * left + 1]),
                   load_dofs=[2 * (n + (n + 1) * n) + 1], load_values=[-1e-3], grid=(n, n, 0)) as p:
        p.set_design(np.random.default_rng(7).uniform(0.3, 1.0, n * n))
        check(p, M.default_opts(rtol=1e-9))


# 72,361 nodes: the last square with rows in registers; 78,961: streamed
@pytest.mark.parametrize("n", [5, 268, 280])
def test_heat_cg_and_bicgstab(n):
    o = M.default_opts(rtol=1e-10, newton_rtol=1e-10, krylov=M.KRYLOV_CG)
    with M.heat_square(n, n) as p:
        T, rep = p.solve(o)
        assert rep.status == 0
        J = csr_at(p, T)
        rhs = np.random.default_rng(8).normal(size=p.n_dofs)
        rhs[p.fixed_dofs] = 0.0
        lam = p.adjoint_solve(T, rhs, M.default_opts(rtol=1e-9, krylov=M.KRYLOV_BICGSTAB))
    assert np.linalg.norm(rhs - J.T @ lam) <= 2e-9 * np.linalg.norm(rhs)


def csr_at(p, X):
    p.residual_and_jacobian(X)
    return csr(p)


def test_rows_longer_than_the_structured_stencil():
    """Ten hexahedra around one edge: 126 columns in the edge's rows, more than a group of
    lanes holds in one round."""
    ns = 10
    t = 2 * np.pi * np.arange(ns) / ns
    ring = np.stack([np.cos(t), np.sin(t)], 1)
    mid = 1.3 * np.stack([np.cos(t + np.pi / ns), np.sin(t + np.pi / ns)], 1)
    xy = np.concatenate([[[0.0, 0.0]], ring, mid])
    coords = np.concatenate([np.c_[xy, np.full(len(xy), z)] for z in (0.0, 1.0)])
    quad = np.array([[0, 1 + i, 1 + ns + i, 1 + (i + 1) % ns] for i in range(ns)])
    conn = np.concatenate([quad, quad + len(xy)], axis=1).astype(np.int32)
    bottom = np.arange(len(xy))
    with M.Problem(M.PHYS_HEX8, coords, conn, M.SIMP_MATERIAL,
                   fixed_dofs=(bottom[:, None] * 3 + np.arange(3)).reshape(-1),
                   load_dofs=[3 * len(xy) + 2], load_values=[-1.0]) as p:
        p.set_design(np.full(ns, 0.7))
        assert np.diff(p.get_csr()[0]).max() == 126
        check(p, M.default_opts(rtol=1e-10))
