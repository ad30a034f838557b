"""Every kernel variant that the U-Net's convolutions can be dispatched to.

The small-grid kernel and the tile kernels sum in the same order, so which of them runs must
not show: a network's output on a box and on a corner of that box that is cut off far
enough away (the output depends on inputs at most 23 voxels off) agree bit for bit, while the
two
grids take different kernels.  Loss and gradients are compared with autograd in 64 bits that rounds
activations and their gradients to BF16 where the network stores them."""
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import parallelpoissonsolver_gb300 as pps

pytestmark = pytest.mark.gpu

REACH = 24   # 5 + 2 * 4 + 4 * 2 = 21, and up to 2 from where a voxel lies in its pooling blocks
DEFAULT = (16, 32, 64)
OTHERS = [(48, 48, 48), (16, 80, 16), (32, 48, 48), (80, 16, 16), (64, 32, 16)]   # 16 to 96 channels, in blocks of 16, 32, 48


def forward(net, x):
    x = x.contiguous()
    out = torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    net.forward(tuple(x.shape), x.data_ptr(), out.data_ptr(), normalize=False)
    return out


#        channels, box, cut extents.  Default: 512-voxel and 16-warp tiles and the tile kernels of
#        all three levels against smaller tiles and the small kernel on the third; then a box
#        of tiles (16, 8 and 4 wide) against the small kernel on every level.
CUTS = [(DEFAULT, (96, 92, 100), (56, 56, 56))]
CUTS += [(c, box, cut) for c in [DEFAULT] + OTHERS
         for box, cut in [((64, 16, 16), (28, 16, 16)), ((128, 16, 8), (28, 16, 8)), ((160, 16, 4), (28, 16, 4)),
                          ((20, 52, 40), (20, 28, 40))]]


@pytest.mark.parametrize("linear", [False, True])
@pytest.mark.parametrize("ch,box,cut", CUTS)
def test_the_kernel_that_runs_does_not_show(gpu, ch, box, cut, linear):
    net = pps.UNet(ch, seed=5, linear=linear)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    x = torch.randn(box, generator=gen, device="cuda")
    whole = forward(net, x)
    assert bool(torch.isfinite(whole).all())
    for high in itertools.product(*[(0,) if c == b else (0, 1) for b, c in zip(box, cut)]):
        part = tuple(slice(b - c, b) if h else slice(0, c) for b, c, h in zip(box, cut, high))
        got = forward(net, x[part])
        keep, there = [], []
        for b, c, h in zip(box, cut, high):   # what no cut face reaches
            n = c if c == b else c - REACH
            keep.append(slice(c - n, c) if h else slice(0, n))
            there.append(slice(b - n, b) if h else slice(0, n))
        assert torch.equal(got[tuple(keep)], whole[tuple(there)]), high
    net.close()


class Bf16(torch.autograd.Function):
    """Rounded to BF16 and kept in 64 bits: the value (if `value`) and its gradient."""

    @staticmethod
    def forward(ctx, x, value):
        return x.to(torch.bfloat16).double() if value else x.clone()

    @staticmethod
    def backward(ctx, g):
        return g.to(torch.bfloat16).double(), None


def stored_forward(layers, x, relu):
    """unet_reference.forward with the roundings of the library: every stored activation, every
    convolution's data gradient, and the sums of gradients where tensors meet.  Returns the
    output and, per layer, the convolution's input and its (unrounded) sums."""
    F = torch.nn.functional
    seen = []

    def conv(i, t, last=False):
        y = F.conv3d(Bf16.apply(t, False), layers[i][0], layers[i][1], padding=1)
        y.retain_grad()
        seen.append((i, t.detach(), y))
        return Bf16.apply(y, False) if last else Bf16.apply(F.relu(y) if relu else y, True)

    def pool(t):
        return Bf16.apply(F.avg_pool3d(t, 2), True)

    def up(t):
        return F.interpolate(t, scale_factor=2, mode="nearest")

    e1 = conv(1, conv(0, x.to(torch.bfloat16).double()[None, None]))
    e2 = conv(3, conv(2, pool(e1)))
    e3 = conv(5, conv(4, pool(e2)))
    d2 = conv(7, conv(6, torch.cat([up(e3), e2], 1)))
    d1 = conv(9, conv(8, torch.cat([up(d2), e1], 1)))
    return conv(10, d1, last=True)[0, 0], seen


def sparse_params(ch, rng, relu):
    """Weights of +-1, two per output channel (half as many as there are input channels to one of
    a few), dealt evenly to the input channels, and small whole biases; with ReLUs more of them
    positive, or nothing would pass eleven layers."""
    import unet_reference as R
    parts = []
    for cin, cout, _ in R.layer_specs(*ch):
        w = np.zeros((27, cin, cout), np.float32)
        per = max(2, cin // (2 * cout))
        order = np.concatenate([rng.permutation(cin) for _ in range(per * cout // cin + 1)])
        for k in range(per * cout):
            tap = 13 if rng.random() < 0.5 else rng.integers(27)   # the deepest level may be one voxel wide
            w[tap, order[k], k // per] = -1.0 if rng.random() < (0.2 if relu else 0.5) else 1.0
        parts += [w.ravel(), rng.integers(-1, 3 if relu else 2, cout).astype(np.float32)]
    return np.concatenate(parts)


def whole_number_case(ch, shape, relu, device):
    """A network, a sample, and everything that its step gives, in 64 bits.  Weights are 0 and
    +-1, input, biases and output error small whole numbers, so every sum of a convolution is
    exact in 32 bits whatever its order (asserted), and the roundings are the library's."""
    import unet_reference as R
    rng = np.random.default_rng(int(np.prod(shape)) + ch[0] + relu)
    params = sparse_params(ch, rng, relu)
    x = torch.from_numpy(rng.integers(-3, 4, shape).astype(np.float32)).to(device)
    err = torch.from_numpy(rng.integers(-1, 3, shape).astype(np.float32)).to(device)
    layers = [(w.detach().to(device).requires_grad_(True), b.detach().to(device).requires_grad_(True))
              for w, b in R.unflatten(params, ch)]
    out, seen = stored_forward(layers, x, relu)
    t = (out.detach() - err.double()).float()
    inv_n = torch.tensor(1.0 / x.numel(), dtype=torch.float64).float().to(device)
    out.backward((2.0 * err * inv_n).double())
    unit = float((2.0 * inv_n).to(torch.bfloat16).double())
    unit = 2.0 ** (np.floor(np.log2(unit)) - 7)   # the lowest bit of a BF16 number of its size
    terms = []
    with torch.no_grad():
        for i, inp, y in seen:
            w, g = layers[i][0].abs(), y.grad
            sums = torch.nn.functional.conv3d(inp.abs(), w, layers[i][1].abs(), padding=1).max()
            back = torch.nn.functional.conv_transpose3d(g.abs(), w, padding=1).max()
            assert float(sums) < 2.0 ** 24 / 64          # values are multiples of 1/64 (two poolings)
            assert i == 0 or float(back) < 2.0 ** 24 * unit / 64
            assert float(g.abs().max()) > 0
            terms.append((i, torch.nn.grad.conv3d_weight(inp.abs(), w.shape, g.abs(), padding=1), g.abs().sum((0, 2, 3, 4)), inp.shape))
    return params, x, t, out.detach(), float((err.double() ** 2).mean()), layers, terms


@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("ch,shape", [(DEFAULT, (68, 68, 84))] +    # the third level in tiles, its data gradients too
                         [(c, s) for c in [DEFAULT] + OTHERS for s in [(8, 12, 16), (20, 24, 36), (48, 16, 8), (96, 16, 4)]])
def test_gradients_of_whole_numbers(gpu, ch, shape, relu):
    """Output and data gradients are exact; a weight's gradient is a 32-bit sum of exact
    products, whose chains (at most half a z plane's steps of 16 voxels, or 64 of a smaller
    plane's) lose at most 2^-23 of the terms a step, and whose few hundred partial sums
    round by 2^-24 each."""
    params, x, t, want, loss_ref, layers, terms = whole_number_case(ch, shape, relu, "cuda")
    net = pps.UNet(ch, seed=1, linear=not relu)
    net.set_params(params)
    out = forward(net, x)
    loss, g = net.gradients(shape, x.data_ptr(), t.data_ptr())
    net.close()
    assert torch.equal(out.double(), want)
    assert abs(loss - loss_ref) <= 1e-12 * loss_ref
    off = 0
    for i, w_terms, b_terms, dims in sorted(terms, key=lambda v: v[0]):
        w, b = layers[i]
        steps = dims[3] * ((dims[4] + 15) // 16)
        tol = max(16, min(64, steps), steps // 2) * 2.0 ** -23 + 600 * 2.0 ** -24

        def flat(v):
            return v.permute(2, 3, 4, 1, 0).reshape(-1).cpu().numpy()

        got = g[off:off + w.numel()].astype(np.float64)
        assert np.all(np.abs(got - flat(w.grad)) <= tol * flat(w_terms)), i
        off += w.numel()
        got = g[off:off + b.numel()].astype(np.float64)
        assert np.all(np.abs(got - b.grad.cpu().numpy()) <= 600 * 2.0 ** -24 * b_terms.cpu().numpy()), i
        off += b.numel()
