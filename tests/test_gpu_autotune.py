"""The autotuner times the kernels that a solve launches."""
import numpy as np
import pytest

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [11, 9])    # three passes; one step and two passes
def test_chebyshev_time_is_that_of_the_launches_of_a_solve(gpu, degree):
    """cheb_us against the launches of a solve that is timed launch by launch.  Where the
    steps run three at a time a launch takes over twice the time of one step's, so a factor
    of 1.5 tells them apart."""
    grid = pps.BlockGrid.cube(256)
    s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(degree), tolerance=1e-10, max_iteration=400, form="mixed", use_graph=False)
    t = s.autotune()
    x, b = grid.new_field(), grid.new_field()
    sl = grid.unknowns()
    b[sl] = np.random.default_rng(0).standard_normal(b[sl].shape)
    assert s(x, b) == pps.OK
    st = s.stats()
    s.close()
    took = 1e6 * st["sweep_seconds"] / st["sweep_launches"]
    assert took / 1.5 <= t["cheb_us"] <= took * 1.5
