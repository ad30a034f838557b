"""The persistent V-cycle batch where its work items take chunks of planes of every length: a few
small problems, many equal ones, and many uneven ones; residuals of all problems, solutions
of the first, the last and one between against the oracle."""
import numpy as np
import pytest

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", [[18] * 6,                 # 4 planes
                                   [20] * 200,               # 8
                                   [30] * 200,               # 16, of 30: the last chunk is shorter
                                   [26] * 200,               # whole columns, one column per thread
                                   [36, 20, 26, 32] * 50])   # columns and quads
def test_every_chunk_length_solves(gpu, oracle, edges):
    grids = [pps.BlockGrid.cube(m) for m in edges]
    rng = np.random.default_rng(len(edges) + edges[0])
    bt = pps.Batch(grids, tolerance=1e-10, inner_tol=1e-5, method="vcycle")
    rhs = []
    for p, g in enumerate(grids):
        b = g.new_field()
        b[g.unknowns()] = rng.standard_normal((edges[p],) * 3)
        rhs.append(b)
        bt.set(p, g.new_field(), b)
    assert bt.solve() == pps.OK, pps.last_error()
    out = [bt.get(p) for p in range(len(edges))]
    bt.close()
    assert max(ps["err_true"] for _, ps in out) <= 1e-10
    for p in (0, len(edges) // 2 + 1, len(edges) - 1):
        want = grids[p].new_field()
        oracle.solve(oracle.cube(edges[p]), oracle.Config(tol=1e-13, maxit=20000, threads=8), want, rhs[p].copy())
        sl = grids[p].unknowns()
        assert np.linalg.norm(out[p][0][sl] - want[sl]) <= 1e-7 * np.linalg.norm(want[sl])
