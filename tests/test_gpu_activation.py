"""Starting some of a batch's designs costs the launches of starting one."""
import numpy as np
import pytest

import mastgpu as M

pytestmark = pytest.mark.gpu


def test_a_subset_starts_with_the_launches_of_one_design():
    rng = np.random.default_rng(51)
    shapes = [(8, 4, 4), (16, 8, 8), (9, 8, 3), (24, 12, 12), (6, 5, 4)]
    des = [dict(nx=s[0], ny=s[1], nz=s[2], rho=rng.uniform(0.2, 1.0, s[0] * s[1] * s[2]), spans=[(0, s[1])])
           for s in shapes]
    # caps that every solve reaches: the same steps whatever takes part
    o = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-12, inner_rtol=1e-6, timeout_s=300.0)
    o.max_iterations, o.max_refinements = 1, 2
    with M.Batch(des) as b:
        b.solve(o, raise_on_error=False)
        counts, results = [], []
        for active in ([1, 0, 0, 0, 0], [0, 0, 0, 1, 0], [1, 0, 1, 0, 1], [0, 1, 1, 0, 1], [1, 1, 1, 1, 1]):
            n0 = M.lib().mg_launch_count()
            _, reps = b.solve(o, active=np.array(active, np.uint8), raise_on_error=False)
            counts.append(M.lib().mg_launch_count() - n0)
            assert all(reps[i].krylov_iterations == 2 for i in range(5) if active[i])
            results.append([b.results(i)[:2] for i in range(5) if active[i]])
    assert len(set(counts)) == 1, counts
    for i, act in ((0, [0, 2, 4]), (1, [1, 2, 4])):
        for (c, dc), k in zip(results[2 + i], act):
            assert np.array_equal(c, results[4][k][0]) and np.array_equal(dc, results[4][k][1])
