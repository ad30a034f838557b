"""The weight and bias gradients' long sums against 64 bits.

With weights that pass channel 0 of every layer on unchanged (identity activations) and an
input and target that are constant on blocks of 4^3, every activation and every output
gradient is known exactly, so the gradients are sums of known products.  All terms have one
sign: an accumulator that truncates then errs in one direction, in proportion to the number
of steps summed in it, and rounding errors of independent sums stay far below that."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu

CH = (16, 32, 64)
SPEC = [(1, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16), (16, 1)]
OFF = np.concatenate([[0], np.cumsum([27 * a * b + b for a, b in SPEC])])


def identity_params():
    p = np.zeros(OFF[-1], np.float32)
    for off, (a, b) in zip(OFF, SPEC):
        p[off + 13 * a * b] = 1.0   # centre tap, channel 0 -> 0 (the upsampled one of a concatenation)
    return p


def shifted(x, tap):
    dz, dy, dx = tap // 9 - 1, (tap // 3) % 3 - 1, tap % 3 - 1
    d, h, w = x.shape
    return torch.nn.functional.pad(x, (1,) * 6)[1 + dz:1 + dz + d, 1 + dy:1 + dy + h, 1 + dx:1 + dx + w]


@pytest.mark.parametrize("shape", [(16, 16, 16), (64, 48, 40), (96, 96, 96), (40, 128, 128), (128, 16, 16)])
def test_gradient_sums_against_64_bits(gpu, shape):
    """Tolerances: a chain of the FP32 accumulator takes at most half of a z plane's steps of 16
    voxels, or up to 64 of a smaller plane's, or one tile's 16; each step loses at most a unit
    in the last place (2^-23) of the running sum, half the chain's sum on average: steps * 2^-24.
    The sums of chains, and those of the bias, round to nearest: up to 1000 of them walk
    1000^(1/2) * 2^-24 = 2e-6."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7)

    def blocks():
        return torch.randint(32, 128, tuple(v // 4 for v in shape), generator=gen, device="cuda").double() / 64

    def fine(v):
        for axis in range(3):
            v = v.repeat_interleave(4, axis)
        return v.float().contiguous()

    a = blocks()
    x, t = fine(a), fine(a - blocks())   # the network's output is x: the gradient has one sign
    net = pps.UNet(CH, seed=1, linear=True)
    net.set_params(identity_params())
    torch.cuda.synchronize()
    _, g = net.gradients(shape, x.data_ptr(), t.data_ptr())
    net.close()
    inv_n = torch.tensor(1.0 / x.numel(), dtype=torch.float64).float().cuda()
    out = (2.0 * (x - t) * inv_n).to(torch.bfloat16).double()
    deep = 64.0 * out[::4, ::4, ::4]     # two sums over 8 equal values each
    for layer, act, grad in ((10, x.double(), out), (5, a, deep)):
        d, h, w = act.shape
        steps = h * ((w + 15) // 16)
        tol = max(16, min(64, steps), steps // 2) * 2.0 ** -24 + 2e-6
        cin, cout = SPEC[layer]
        for tap in range(27):
            terms = shifted(act, tap) * grad
            got = float(g[OFF[layer] + tap * cin * cout])
            assert abs(got - float(terms.sum())) <= tol * float(terms.abs().sum()), (layer, tap)
        bias = float(g[OFF[layer] + 27 * cin * cout])
        assert abs(bias - float(grad.sum())) <= 2e-6 * float(grad.abs().sum()), layer
