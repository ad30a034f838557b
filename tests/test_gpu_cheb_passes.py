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


DOT_SHAPES = [(3, 1, 1), (126, 7, 9), (127, 8, 12), (128, 6, 13), (256, 33, 5), (257, 3, 40), (30, 62, 21), (517, 2, 70)]


@pytest.mark.parametrize("n", DOT_SHAPES)
def test_x_vectorised_dots_match_the_one_column_tiles(gpu, n):
    """BiCGSTAB's stencils on float4s against the one-column kernels, where rows end inside
    a float4, a warp or a block.  Per point the arithmetic is the same and the double-float
    sums agree to 1e-12; an FP32 scalar that rounds the other way (6e-8) moves the residuals
    of three steps by far less than 1e-5 of the first."""
    grid = pps.BlockGrid(npglobal=tuple(v + 2 for v in n), ds=(0.03, 0.035, 0.025))
    b = grid.new_field()
    sl = grid.unknowns()
    b[sl] = np.random.default_rng(3).standard_normal(b[sl].shape)
    runs = []
    for cx in (4, 1):
        s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(8), tolerance=1e-12, max_iteration=3, form="mixed")
        s.set_tuning({**s.tuning(), "cheb_cx": cx})
        x = grid.new_field()
        s(x, b.copy())
        runs.append((s.history(), x))
        s.close()
    (h4, x4), (h1, x1) = runs
    k = min(len(h4), len(h1))
    assert k >= 2 and np.all(np.isfinite(h4[:k]))
    assert np.max(np.abs(h4[:k] - h1[:k])) <= 1e-5 * h1[0]
    assert np.linalg.norm(x4 - x1) <= 1e-4 * np.linalg.norm(x1)
