"""Tile numbers of the longest sides that the matrix-free form accepts: the tensor-core operator's
columns are seven nodes wide, so a side of 262,000 elements has more of them than a signed 16-bit
number can count.  A number that wrapped would put a column in front of its problem's vectors."""
import os
import subprocess

import numpy as np
import pytest

import mastgpu as M
import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "mast-multiphysics_gb300", "csrc")


def test_the_last_column_of_the_longest_side_keeps_its_number():
    out = os.path.join(HERE, "cpp", "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "tile_numbers_host")
    subprocess.run([M._nvcc(), "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-x", "cu", "-I", CSRC,
                    "-I", os.path.join(HERE, "..", "include"), os.path.join(HERE, "cpp", "tile_numbers_host.cpp"),
                    "-o", exe], check=True)
    lines = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]
    assert len(lines) == 3
    for line in lines:
        name, want, stored = line.split()
        assert int(want) == int(stored), line


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(M.MIXED_TF32X3, 2e-5), (M.OPERATOR_FACTORED_FP32, 2e-6)])
def test_operator_on_a_beam_of_230000_elements(precision, tol):
    """The first side whose columns pass the signed range, against the element products (relative
    to the largest entry, the bar of the operators against the assembled form)."""
    nx = 230000
    rng = np.random.default_rng(61)
    with M.simp_cantilever(nx, 1, 1) as p:
        p.set_design(np.ones(nx))
        x = rng.uniform(-1.0, 1.0, p.n_dofs)
        x[p.fixed_dofs] = 0.0
        y = p.matfree_apply(x, precision)
        Ke = O.hex8_internal(p.coords[p.conn[0]], 1.0, 0.3)[1]
        ue = x.reshape(-1, 3)[p.conn].transpose(0, 2, 1).reshape(nx, 24)  # var-blocked
        ye = (ue @ Ke.T).reshape(nx, 3, 8).transpose(0, 2, 1)
        ref = np.zeros((p.n_nodes, 3))
        for a in range(8):
            np.add.at(ref, p.conn[:, a], ye[:, a])
        ref = ref.reshape(-1)
        ref[p.fixed_dofs] = 0.0
    assert np.abs(y - ref).max() / np.abs(ref).max() < tol
