"""pps_apply_operator_noalloc call after call on its one scratch array: grids of one block and of
thousands queued back to back without a wait in between, and calls after others that
overlapped.  Each energy is compared with the same sum taken on the host in FP64 (the
tolerance of the other tests of this entry point, 1e-12 of the terms' magnitudes)."""
import numpy as np
import pytest

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu

#        unknowns (x, y, z)
SIZES = [(1, 1, 1), (200, 180, 96), (5, 3, 2), (64, 48, 80), (33, 9, 17), (257, 130, 60), (31, 7, 1)]


class Call:
    """One grid's buffers and the energy the call has to give."""

    def __init__(self, torch, n, seed):
        self.grid = pps.BlockGrid(npglobal=tuple(v + 2 for v in n), ds=(0.05, 0.07, 0.04) if seed % 2 else (0.05,) * 3)
        u = np.zeros(self.grid.shape)
        sl = self.grid.unknowns()
        u[sl] = np.random.default_rng(seed).standard_normal(u[sl].shape)
        au = np.zeros_like(u[sl])
        for axis, d in enumerate((2, 1, 0)):
            lo, hi = list(sl), list(sl)
            lo[axis], hi[axis] = (slice(sl[axis].start + o, sl[axis].stop + o) for o in (-1, 1))
            au += (u[tuple(lo)] - 2.0 * u[sl] + u[tuple(hi)]) / self.grid.ds[d] ** 2
        self.want, self.scale = float(np.sum(u[sl] * au)), float(np.sum(np.abs(u[sl] * au)))
        self.u = torch.from_numpy(u).cuda()
        self.out = torch.zeros_like(self.u)
        self.energy = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")

    def queue(self, stream, energy=None):
        st = pps.apply_operator_noalloc(self.grid, self.u.data_ptr(), self.out.data_ptr(),
                                        self.energy.data_ptr() if energy is None else energy, stream.cuda_stream)
        assert st == pps.OK, pps.last_error()

    def right(self):
        return abs(self.energy.item() - self.want) <= 1e-12 * self.scale


def test_calls_queued_back_to_back_give_their_own_energies(gpu):
    torch = pytest.importorskip("torch")
    calls = [Call(torch, n, k) for k, n in enumerate(SIZES * 3)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for c in calls:
        c.queue(stream)
    torch.cuda.synchronize()
    assert [c.grid.npglobal for c in calls if not c.right()] == []


def test_calls_after_overlapping_ones_are_right(gpu):
    """Calls that overlap on the GPU race for the scratch (their energies are undefined, the
    accesses stay inside it); what follows once they ended must not notice."""
    torch = pytest.importorskip("torch")
    calls = [Call(torch, n, k) for k, n in enumerate(SIZES)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(30):
        for c, d in zip(calls, calls[::-1]):
            c.queue(streams[0])
            d.queue(streams[1])
    torch.cuda.synchronize()
    for c in calls:
        c.energy.fill_(float("nan"))
    torch.cuda.synchronize()
    for c in calls:
        c.queue(streams[0])
    torch.cuda.synchronize()
    assert [c.grid.npglobal for c in calls if not c.right()] == []


@pytest.mark.parametrize("offset", [1, 2, 4, 7])
def test_the_energy_may_lie_at_any_address(gpu, offset):
    torch = pytest.importorskip("torch")
    for k, n in enumerate([(1, 1, 1), (64, 48, 80)]):
        c = Call(torch, n, k)
        room = torch.full((24,), 0xA5, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        c.queue(torch.cuda.current_stream(), room.data_ptr() + offset)
        torch.cuda.synchronize()
        got = room.cpu().numpy()
        value = got[offset:offset + 8].copy().view(np.float64)[0]
        assert abs(value - c.want) <= 1e-12 * c.scale
        assert np.all(got[:offset] == 0xA5) and np.all(got[offset + 8:] == 0xA5)
