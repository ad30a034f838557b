"""The buffers of the MIXED form's Chebyshev applications: the three-step passes keep the two
steps they leave in the solver's three work buffers and the output field, so they need no
device memory beyond the one-step kernels', and values of the output field off the unknowns
(boundary nodes, guards: the caller's) never reach a result."""
import gc

import numpy as np
import pytest

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu


# degree - 2 steps: passes of three, 0, 1 or 2 left over (an even and an odd number of passes)
@pytest.mark.parametrize("degree", [5, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 19])
#                                       8-byte quads (one tile along x, several along y), 16-byte quads (several
#                                       along both), rows of 8 lanes; one that runs in passes up to degree 7 alone
@pytest.mark.parametrize("n", [(62, 50, 40), (252, 40, 30), (30, 80, 86), (64, 32, 33)])
def test_passes_ignore_the_output_field_off_the_unknowns(gpu, oracle, n, degree):
    """Against the oracle with the one-step FP32 preconditioner's tolerance (2e-5)."""
    npg, ds = tuple(v + 2 for v in n), (0.03, 0.035, 0.025)
    grid = pps.BlockGrid(npglobal=npg, ds=ds)
    rng = np.random.default_rng(degree)
    B, X = rng.standard_normal(grid.shape), 1e3 * rng.standard_normal(grid.shape)
    s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(degree), form="mixed")
    got = s.apply_preconditioner(B.copy(), X.copy())
    again = s.apply_preconditioner(B.copy(), np.zeros_like(X))
    s.close()
    cfg = oracle.Config(cheb_degree=degree, cheb_eps=1e-4, rescale_min=500.0, rescale_max=1.0 - 1e-4)
    want = oracle.cheb_apply(oracle.Grid(npg, ds, (0.0, 0.0, 0.0), (0,) * 6), cfg, B.copy())
    sl = grid.unknowns()
    assert np.linalg.norm(got[sl] - want[sl]) <= 2e-5 * np.linalg.norm(want[sl])
    assert np.array_equal(got[sl], again[sl])
    off = np.ones(grid.shape, bool)
    off[sl] = False
    assert np.array_equal(got[off], X[off].astype(np.float32).astype(np.float64))


@pytest.mark.parametrize("bcs", [(0,) * 6, (0, 1) * 3])
def test_a_mixed_solver_takes_60_bytes_a_point(gpu, bcs):
    """x and b in FP64 and eleven FP32 fields; 2 bytes a point cover the small buffers and the
    rounding of 13 allocations to 2 MB."""
    torch = pytest.importorskip("torch")
    grid = pps.BlockGrid(npglobal=(256, 256, 256), ds=(0.03, 0.03, 0.03), bcs=bcs)
    points = int(np.prod(grid.shape))

    def make():
        s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(11), form="mixed")
        torch.cuda.synchronize()
        return s, torch.cuda.mem_get_info()[0]

    make()[0].close()                     # the context's and the kernels' own memory
    gc.collect()                          # nor what earlier tests left behind
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s, after = make()
    s.close()
    assert 60 * points <= before - after <= 62 * points
