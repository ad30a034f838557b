"""The MIXED form's float4 kernels on grids that take them: rows of npglobal[0] + 2 = 4k
points.  The Neumann variants of the Chebyshev sweeps (quads stored with their mirrored ghost
points), the stencils with sums on rows that end anywhere in a block, and the 16-byte
three-step passes over several tiles along y."""
import numpy as np
import pytest

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu

FACES = {"lower x": (1, 0, 0, 0, 0, 0), "upper x": (0, 1, 0, 0, 0, 0), "both x": (1, 1, 0, 0, 0, 0),
         "y and z": (0, 0, 1, 0, 0, 1), "uppers": (0, 1, 0, 1, 0, 1), "lowers": (1, 0, 1, 0, 1, 0)}


def config(oracle, degree):
    return oracle.Config(cheb_degree=degree, cheb_eps=1e-4, rescale_min=500.0, rescale_max=1.0 - 1e-4)


@pytest.mark.parametrize("degree", [3, 4, 8])
@pytest.mark.parametrize("faces", list(FACES))
@pytest.mark.parametrize("npx", [6, 14, 34, 130, 258])
def test_float4_sweeps_with_neumann_faces_match_the_oracle(gpu, oracle, npx, faces, degree):
    """Tolerance of the one-step FP32 preconditioner (2e-5)."""
    npg, ds, bcs = (npx, 11, 13), (0.03, 0.035, 0.025), FACES[faces]
    grid = pps.BlockGrid(npglobal=npg, ds=ds, bcs=bcs)
    assert grid.shape[2] % 4 == 0
    B = np.random.default_rng(degree).standard_normal(grid.shape)
    s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(degree), form="mixed")
    assert s.tuning()["cheb_cx"] == 4
    got = s.apply_preconditioner(B.copy())
    s.close()
    want = oracle.cheb_apply(oracle.Grid(npg, ds, (0.0, 0.0, 0.0), bcs), config(oracle, degree), B.copy())
    sl = grid.unknowns()
    assert np.linalg.norm(got[sl] - want[sl]) <= 2e-5 * np.linalg.norm(want[sl])


@pytest.mark.parametrize("n", [(4, 1, 1), (4, 70, 3), (60, 9, 9), (124, 8, 12), (132, 6, 13), (252, 33, 5), (260, 3, 40), (516, 2, 70)])
@pytest.mark.parametrize("faces", [None, "lower x", "upper x", "uppers"])
def test_sums_on_float4_rows_match_the_one_column_tiles(gpu, n, faces):
    """Per point the arithmetic is the same and the double-float sums agree to 1e-12; an FP32
    scalar that rounds the other way (6e-8) moves the residuals of three steps by far less
    than 1e-5 of the first."""
    bcs = FACES[faces] if faces else (0,) * 6
    npg = tuple(n[a] + 2 if a == 0 else n[a] + 2 - bcs[2 * a] - bcs[2 * a + 1] for a in range(3))
    npg = tuple(max(3, v) for v in npg)
    grid = pps.BlockGrid(npglobal=npg, ds=(0.03, 0.035, 0.025), bcs=bcs)
    assert grid.shape[2] % 4 == 0
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


@pytest.mark.parametrize("faces", list(FACES))
def test_mixed_solves_with_neumann_faces_on_float4_rows(gpu, oracle, faces):
    """Against the oracle's solution: residuals of 1e-10 and of 1e-13 on a grid whose operator
    is far better conditioned than 1e3."""
    npg, ds, bcs = (34, 20, 17), (0.1, 0.1, 0.1), FACES[faces]
    grid = pps.BlockGrid(npglobal=npg, ds=ds, bcs=bcs)
    b = grid.new_field()
    sl = grid.unknowns()
    b[sl] = np.random.default_rng(8).standard_normal(b[sl].shape)
    s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(11), tolerance=1e-10, max_iteration=2000, form="mixed")
    x = grid.new_field()
    assert s(x, b.copy()) == pps.OK
    s.close()
    want = grid.new_field()
    oracle.solve(oracle.Grid(npg, ds, (0.0, 0.0, 0.0), bcs), oracle.Config(tol=1e-13, maxit=20000, threads=8), want, b.copy())
    assert np.linalg.norm(x[sl] - want[sl]) <= 1e-6 * np.linalg.norm(want[sl])


@pytest.mark.parametrize("degree", [5, 9, 10, 11])
@pytest.mark.parametrize("n", [(252, 47, 25), (500, 40, 16), (60, 95, 24), (252, 18, 50)])   # 16-byte quads, tiles along y (and x)
def test_16_byte_passes_over_several_tiles_match_the_oracle(gpu, oracle, n, degree):
    npg, ds = tuple(v + 2 for v in n), (0.03, 0.035, 0.025)
    grid = pps.BlockGrid(npglobal=npg, ds=ds)
    assert grid.shape[2] % 4 == 0
    B = np.random.default_rng(degree).standard_normal(grid.shape)
    s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(degree), form="mixed")
    got = s.apply_preconditioner(B.copy())
    s.close()
    want = oracle.cheb_apply(oracle.Grid(npg, ds, (0.0, 0.0, 0.0), (0,) * 6), config(oracle, degree), B.copy())
    sl = grid.unknowns()
    assert np.linalg.norm(got[sl] - want[sl]) <= 2e-5 * np.linalg.norm(want[sl])


@pytest.mark.parametrize("degree", [8, 9, 10, 11])
@pytest.mark.parametrize("n", [(62, 32, 66),      # 16 lanes a row
                               (30, 62, 113),     # 8 lanes a row, the last quad half full
                               (128, 25, 41),     # a row is exactly 32 quads from its first unknown
                               (130, 19, 52),     # two tiles along x, ragged
                               (250, 18, 29),     # 8-byte quads, three tiles
                               (252, 7, 150)])    # fewer rows than a tile
def test_several_passes_on_ragged_tiles_match_the_oracle(gpu, oracle, n, degree):
    npg, ds = tuple(v + 2 for v in n), (0.03, 0.035, 0.025)
    grid = pps.BlockGrid(npglobal=npg, ds=ds)
    B = np.random.default_rng(degree).standard_normal(grid.shape)
    s = pps.BiCGSTAB(grid, pps.ChebyshevIteration(degree), form="mixed")
    got = s.apply_preconditioner(B.copy())
    s.close()
    want = oracle.cheb_apply(oracle.Grid(npg, ds, (0.0, 0.0, 0.0), (0,) * 6), config(oracle, degree), B.copy())
    sl = grid.unknowns()
    assert np.linalg.norm(got[sl] - want[sl]) <= 2e-5 * np.linalg.norm(want[sl])
