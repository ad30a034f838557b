"""Building-block calls leave a solver's work fields as its solves expect them: zero off the
unknowns, whatever the caller's arrays hold there (boundary nodes, guards)."""
import numpy as np
import pytest

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bcs", [(0,) * 6, (0, 1) * 3])
@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [(20, 18, 22), (64, 32, 33)])
def test_preconditioner_is_the_same_after_an_operator_call(gpu, n, form, bcs):
    grid = pps.BlockGrid(npglobal=tuple(v + 2 for v in n), ds=(0.03, 0.03, 0.03), bcs=bcs)
    rng = np.random.default_rng(4)
    B = grid.new_field()
    sl = grid.unknowns()
    B[sl] = rng.standard_normal(B[sl].shape)
    u = 1e3 * rng.standard_normal(grid.shape)
    s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(11), form=form)
    first = s.apply_preconditioner(B.copy())
    s.apply_operator(u, np.zeros_like(u))
    second = s.apply_preconditioner(B.copy())
    s.close()
    assert np.array_equal(first[sl], second[sl])
