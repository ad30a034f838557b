"""The three-steps-a-pass FP32 Chebyshev kernel (MIXED form, 64 K unknowns and more)
against the oracle, at the sizes where its tiles end raggedly and at the degrees whose
step count leaves none, one or two steps to the one-step kernels (chebyshevIteration.hpp:
48-140).  B holds values off the unknowns too: the first step reads them as stored.  The
tolerance is the one-step FP32 preconditioner's (2e-5)."""
import numpy as np
import pytest

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu

#        unknowns (x, y, z)
SHAPES = [(64, 32, 33),      # 16 lanes a row
          (30, 62, 71),      # 8 lanes a row, the last quad half full
          (128, 25, 24),     # a row is exactly 32 quads from its first unknown
          (130, 19, 40),     # two tiles along x, ragged
          (250, 18, 17),     # 16-byte quads from x = 0, three tiles
          (252, 7, 40),      # fewer rows than a tile
          (129, 25, 24)]     # odd rows: the one-step kernels


@pytest.mark.parametrize("degree", [5, 6, 7, 8, 11])
@pytest.mark.parametrize("n", SHAPES)
def test_three_step_passes_match_the_oracle(gpu, oracle, n, degree):
    npg, ds = tuple(v + 2 for v in n), (0.03, 0.035, 0.025)
    grid = pps.BlockGrid(npglobal=npg, ds=ds)
    B = np.random.default_rng(degree).standard_normal(grid.shape)
    s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(degree), form="mixed")
    got = s.apply_preconditioner(B.copy())
    s.close()
    cfg = oracle.Config(cheb_degree=degree, cheb_eps=1e-4, rescale_min=500.0, rescale_max=1.0 - 1e-4)
    want = oracle.cheb_apply(oracle.Grid(npg, ds, (0.0, 0.0, 0.0), (0,) * 6), cfg, B.copy())
    sl = grid.unknowns()
    assert np.linalg.norm(got[sl] - want[sl]) <= 2e-5 * np.linalg.norm(want[sl])
