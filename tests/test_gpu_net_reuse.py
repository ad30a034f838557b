"""A network that works for a solver and elsewhere in between: other extents, training and another
activation replace its buffers or what its layers do, and the solver's captured iterations,
kept from solve to solve, must not outlive either."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu


def solver(net, form):
    s = pps.FlexibleCG(pps.BlockGrid.cube(32), pps.ChebyshevIteration(11), tolerance=1e-10, max_iteration=60, form=form)
    s.set_learned(net, 1, 1.0, pps.LEARNED_PRECONDITIONER | pps.LEARNED_NO_FALLBACK)
    s.set_learned_cycle(5, 4, 8.0)
    return s


def solve(s, b):
    x = np.zeros_like(b)
    s(x, b.copy())
    return x, s.history()


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_a_solver_sees_what_its_network_did_in_between(gpu, form):
    net = pps.UNet((16, 32, 64), seed=2, linear=True)
    grid = pps.BlockGrid.cube(32)
    b = grid.new_field()
    b[grid.unknowns()] = np.random.default_rng(0).standard_normal((32,) * 3)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    s = solver(net, form)
    x1, h1 = solve(s, b)
    filled = []

    def use(m, train):
        """The network on m^3; then what the device hands out next is filled with junk."""
        u, t = (torch.randn((m,) * 3, generator=gen, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        if train:
            net.gradients((m,) * 3, u.data_ptr(), t.data_ptr())
        else:
            net.forward((m,) * 3, u.data_ptr(), torch.empty_like(u).data_ptr())
        filled.append(torch.full((1 << 22,), float("nan"), device="cuda"))
        torch.cuda.synchronize()

    for m, train in ((24, False), (16, True), (8, True), (16, False)):   # the solver's is 16^3
        use(m, train)
        x, h = solve(s, b)
        assert np.array_equal(h, h1) and np.array_equal(x, x1), (m, train)
    # another activation: as a fresh solver with it
    assert pps.load().pps_unet_set_activation(net.handle, 0) == pps.OK
    x2, h2 = solve(s, b)
    fresh = solver(net, form)
    x3, h3 = solve(fresh, b)
    fresh.close()
    s.close()
    net.close()
    assert np.array_equal(h2, h3) and np.array_equal(x2, x3) and not np.array_equal(h2, h1)
