"""The work that users of this framework have it do, as cases that can be timed.

Each case is one call (or one training step) through the package's public entry points:

* operator  -- A u and sum u*(A u) on device fields, queued on the caller's stream
               (apply_operator_noalloc), as an outer solver or a time stepper calls it;
* solve     -- one Poisson solve by the reference's methods (BiCGSTAB or CG with the
               Chebyshev preconditioner, FP64 or mixed precision, Dirichlet and Neumann
               faces), on device fields or on host arrays;
* learned   -- one solve by flexible CG whose preconditioner is a multigrid V-cycle with
               the U-Net on its coarsest level;
* batch     -- many independent grids of uneven size solved together;
* forward, gradients, train -- the U-Net's inference, its loss and gradients, and one
               Adam step.

Right-hand sides are those of the benchmark workloads: Gaussian random fields with
P(k) ~ k^-2 and unit RMS, and (batches, training) sums of 1-8 Gaussian blobs.
"""
import functools
import math

import numpy as np
import torch
import torch.nn.functional as F

import parallelpoissonsolver_gb300 as pps
from parallelpoissonsolver_gb300 import learned, workloads

DEV = "cuda"
CHANNELS = (16, 32, 64)
LAYERS = ((1, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16), (16, 1))
ADAM = (0.9, 0.999, 1e-8)


def listed():
    return [
        # the operator on a small box and on a large ragged one (a time stepper, an outer Krylov loop)
        {"name": "operator_64x48x80", "kind": "operator", "nx": 64, "ny": 48, "nz": 80},
        {"name": "operator_401x250x317", "kind": "operator", "nx": 401, "ny": 250, "nz": 317},
        # the first solve a user of the reference tries: 64^3, its default method, host arrays
        {"name": "fp64_host_64", "kind": "solve", "krylov": "bicgstab", "form": "fp64", "nx": 64, "ny": 64, "nz": 64,
         "neumann": False, "tol": 1e-10, "host": True},
        # the reference's one recorded run: 128 x 128 x 256, Dirichlet and Neumann faces in turn, 1e-8
        {"name": "fp64_neumann_128x128x256", "kind": "solve", "krylov": "bicgstab", "form": "fp64", "nx": 127,
         "ny": 127, "nz": 255, "neumann": True, "tol": 1e-8, "host": False},
        # the reference's method in mixed precision at a production size
        {"name": "mixed_256", "kind": "solve", "krylov": "bicgstab", "form": "mixed", "nx": 256, "ny": 256,
         "nz": 256, "neumann": False, "tol": 1e-10, "host": False},
        # the learned preconditioner in FP64 at 128^3 (the training and evaluation grid)
        {"name": "learned_fp64_128", "kind": "learned", "form": "fp64", "net": 16, "coarsen": 3},
        # the benchmark's headline solve
        {"name": "learned_mixed_512", "kind": "learned", "form": "mixed", "net": 16, "coarsen": 5},
        # the batched workload: 256 uneven cubes in one persistent launch
        {"name": "batch_vcycle_256", "kind": "batch", "method": "vcycle", "count": 256, "edges": "32,48,64,96,128"},
        # the reference's method on a batch whose edges the V-cycle does not take
        {"name": "batch_bicgstab_24", "kind": "batch", "method": "bicgstab", "count": 24, "edges": "17,30,33,50,63"},
        # one step of the network's training (20,000 and more of them make a network)
        {"name": "train_16", "kind": "train", "nx": 16, "ny": 16, "nz": 16, "linear": True, "lr": 2e-4},
        # loss and gradients on a larger, ragged grid with ReLU layers (an outer optimiser, data-parallel training)
        {"name": "gradients_64x48x40", "kind": "gradients", "nx": 64, "ny": 48, "nz": 40, "linear": False},
        # the network as a solver of its own on the 128^3 grid
        {"name": "forward_128", "kind": "forward", "nx": 128, "ny": 128, "nz": 128, "linear": False},
    ]


def _size(rng, lo, hi, multiple=1):
    return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["operator", "solve", "solve", "learned", "batch", "train", "gradients", "forward"])
    c = {"kind": kind}
    if kind == "operator":
        c.update(nx=_size(rng, 16, 420), ny=_size(rng, 16, 320), nz=_size(rng, 16, 320))
    elif kind == "solve":
        form = rng.choice(["fp64", "mixed"])
        top = 110 if form == "fp64" else 200
        c.update(krylov=rng.choice(["bicgstab", "bicgstab", "cg"]), form=form, nx=_size(rng, 24, top),
                 ny=_size(rng, 24, top), nz=_size(rng, 24, top), neumann=rng.random() < 0.25,
                 tol=rng.choice([1e-8, 1e-10]), stretch=rng.choice([1.0, 1.0, 1.0, 1.25]))
        c["host"] = rng.random() < 0.25 and c["nx"] * c["ny"] * c["nz"] < 100 ** 3
    elif kind == "learned":
        form = rng.choice(["fp64", "mixed"])
        c.update(form=form, net=rng.choice([12, 16, 20]), coarsen=rng.randint(1, 3 if form == "fp64" else 4))
    elif kind == "batch":
        method = rng.choice(["vcycle", "bicgstab"])
        edges = [32, 40, 48, 64, 80, 96, 128] if method == "vcycle" else list(range(16, 72))
        c.update(method=method, count=_size(rng, 4, 200 if method == "vcycle" else 40),
                 edges=",".join(str(e) for e in sorted(rng.sample(edges, rng.randint(2, 5)))))
    else:
        top = {"train": 40, "gradients": 80, "forward": 128}[kind]
        c.update(nx=_size(rng, 8, top, 4), ny=_size(rng, 8, top, 4), nz=_size(rng, 8, top, 4),
                 linear=rng.random() < 0.5)
        if kind == "train":
            c["lr"] = rng.choice([1e-4, 2e-4])
    return c


# ---------------------------------------------------------------- grids and right-hand sides

def _grid(case):
    """The box of a case: nx, ny, nz unknowns per axis, spacings equal but for `stretch` times
    the others along z, Dirichlet faces, or Dirichlet at the lower and Neumann at the upper face of every axis."""
    n = (case["nx"], case["ny"], case["nz"])
    neumann = bool(case.get("neumann", False))
    h = 0.1 if neumann else 1.0 / (max(n) + 1)
    return pps.BlockGrid(npglobal=tuple(v + (1 if neumann else 2) for v in n), ds=(h, h, h * case.get("stretch", 1.0)),
                         bcs=(0, 1) * 3 if neumann else (0,) * 6)


def _learned_grid(case):
    return pps.BlockGrid.cube(case["net"] << case["coarsen"])


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _random_field(shape, gen):
    """Unit-RMS Gaussian random field with P(k) ~ k^-2 on (nz, ny, nx) points."""
    spectrum = torch.fft.rfftn(torch.randn(shape, generator=gen, dtype=torch.float64, device=DEV))
    k = [torch.fft.fftfreq(shape[a], d=1.0 / shape[a], dtype=torch.float64, device=DEV) for a in (0, 1)]
    k.append(torch.fft.rfftfreq(shape[2], d=1.0 / shape[2], dtype=torch.float64, device=DEV))
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    spectrum *= k2 ** -0.5
    spectrum[0, 0, 0] = 0.0
    f = torch.fft.irfftn(spectrum, s=shape)
    return f / torch.sqrt(torch.mean(f * f))


def _blobs(m, gen):
    """A sum of 1-8 Gaussian blobs on m^3 points of the unit cube."""
    count = int(torch.randint(1, 9, (1,), generator=gen, device=DEV))
    c = torch.arange(1, m + 1, dtype=torch.float64, device=DEV) / (m + 1)
    centre = 0.2 + 0.6 * torch.rand((3, count, 1), generator=gen, dtype=torch.float64, device=DEV)
    width = 0.02 + 0.08 * torch.rand((1, count, 1), generator=gen, dtype=torch.float64, device=DEV)
    a = torch.randn((count,), generator=gen, dtype=torch.float64, device=DEV)
    gz, gy, gx = torch.exp(-((c - centre) ** 2) / (2 * width * width))
    return torch.einsum("b,bz,by,bx->zyx", a, gz, gy, gx)


def _padded(grid, values):
    b = torch.zeros(grid.shape, dtype=torch.float64, device=DEV)
    b[grid.unknowns()] = values
    return b


def _unknown_shape(grid):
    return tuple(s.stop - s.start for s in grid.unknowns())


def _rhs(grid, seed):
    return _padded(grid, -_random_field(_unknown_shape(grid), _generator(seed)))


def _batch_edges(case, seed):
    edges = [int(e) for e in case["edges"].split(",")]
    picked = np.random.default_rng(3).choice(edges, case["count"])   # the sizes are the case's, not the seed's
    return [int(e) for e in picked]


class _DeviceField:
    """A device field of the library, for torch.as_tensor."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": "<f8",
                                         "strides": None, "version": 3}


# ---------------------------------------------------------------- the network

def _net_forward(weights, x, linear):
    """The U-Net on (n, 1, z, y, x) by plain torch operations."""
    act = (lambda t: t) if linear else torch.relu

    def conv(i, t):
        w, b = weights[i]
        return F.conv3d(t, w, b, padding=1)

    def pool(t):
        n, c, d, h, w = t.shape
        return t.reshape(n, c, d // 2, 2, h // 2, 2, w // 2, 2).mean((3, 5, 7))

    def up(t):
        n, c, d, h, w = t.shape
        return t[:, :, :, None, :, None, :, None].expand(n, c, d, 2, h, 2, w, 2).reshape(n, c, 2 * d, 2 * h, 2 * w)

    e1 = act(conv(1, act(conv(0, x))))
    e2 = act(conv(3, act(conv(2, pool(e1)))))
    e3 = act(conv(5, act(conv(4, pool(e2)))))
    d2 = act(conv(7, act(conv(6, torch.cat([up(e3), e2], 1)))))
    d1 = act(conv(9, act(conv(8, torch.cat([up(d2), e1], 1)))))
    return conv(10, d1)


def _unflatten(flat, dtype):
    out, off = [], 0
    for cin, cout in LAYERS:
        n = 27 * cin * cout
        w = torch.from_numpy(flat[off:off + n]).reshape(3, 3, 3, cin, cout).permute(4, 3, 0, 1, 2)
        b = torch.from_numpy(flat[off + n:off + n + cout])
        out.append((w.to(DEV, dtype).contiguous().requires_grad_(True), b.to(DEV, dtype).requires_grad_(True)))
        off += n + cout
    return out


def _flatten(pairs):
    parts = []
    for w, b in pairs:
        parts += [w.permute(2, 3, 4, 1, 0).reshape(-1), b.reshape(-1)]
    return torch.cat(parts)


def _initial_params(seed):
    """He-scaled weights and small biases, as a network in training has them."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, (cin, cout) in enumerate(LAYERS):
        last = i == len(LAYERS) - 1
        parts.append(rng.standard_normal(27 * cin * cout) * math.sqrt(2.0 / (27 * cin)) * (0.1 if last else 1.0))
        parts.append(rng.standard_normal(cout) * 0.02)
    return np.concatenate(parts).astype(np.float32)


@functools.lru_cache(maxsize=None)
def _trained(n, coarsen):
    """A linear U-Net trained for the coarsest level operator of `coarsen` coarsenings on
    n^3: (flat parameters, output scale).  Trained once per process by plain torch, so
    that every version of the library is given the same weights."""
    data = learned.make_dataset_batch(n, 10000, 1024, coarsen)
    scale = learned.fit_scale(data)
    b = torch.stack([p[0] for p in data])[:, None]
    u = torch.stack([p[1] for p in data])[:, None]
    rms = torch.sqrt(torch.mean(b * b, dim=(1, 2, 3, 4), keepdim=True))
    b, u = b / rms, u / (rms * scale)
    weights = _unflatten(_initial_params(1), torch.float32)
    flat = [t for pair in weights for t in pair]
    order = np.random.default_rng(2)
    steps, batch, lr = 700, 16, 3e-3
    opt = torch.optim.Adam(flat, lr=lr, foreach=True)
    with torch.backends.cudnn.flags(enabled=True, benchmark=False, deterministic=True, allow_tf32=False):
        for k in range(steps):
            for group in opt.param_groups:
                group["lr"] = lr * min(1.0, (k + 1) / 40) * 0.05 ** (k / steps)
            pick = torch.from_numpy(order.choice(len(data), batch, replace=False)).to(DEV)
            opt.zero_grad(set_to_none=True)
            loss = torch.mean((_net_forward(weights, b[pick], True) - u[pick]) ** 2)
            loss.backward()
            torch.nn.utils.clip_grad_norm_(flat, 1.0)
            opt.step()
    return _flatten([(w.detach(), c.detach()) for w, c in weights]).cpu().numpy(), scale


def _net_sample(case, seed):
    """An input of unit RMS and a smoother target of the same grid, as training pairs are."""
    gen = _generator(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    x = _random_field(shape, gen)
    t = _random_field(shape, gen) * 0.1 + 0.5 * torch.roll(x, 1, 2)
    return x.float().contiguous(), t.float().contiguous()


# ---------------------------------------------------------------- preparation

def prepare(case, seed):
    kind = case["kind"]
    if kind == "operator":
        grid = _grid(case)
        s = {"grid": grid, "u": _rhs(grid, seed), "energy": torch.zeros(1, dtype=torch.float64, device=DEV)}
        s["out"] = torch.zeros_like(s["u"])
    elif kind == "solve":
        grid = _grid(case)
        method = pps.BiCGSTAB if case["krylov"] == "bicgstab" else pps.BaseCG
        s = {"solver": method(grid, pps.ChebyshevIteration(11), tolerance=case["tol"], max_iteration=20000,
                              form=case["form"]), "b": _rhs(grid, seed)}
        if case["host"]:
            s["b"] = s["b"].cpu().numpy()
            s["x"] = grid.new_field()
        else:
            s["x"] = torch.zeros_like(s["b"])
    elif kind == "learned":
        grid = _learned_grid(case)
        n, k = case["net"], case["coarsen"]
        params, scale = _trained(n, k)
        net = pps.UNet(CHANNELS, seed=1, linear=True)
        net.set_params(params)
        gain = scale * ((2 ** k / ((n << k) + 1)) * (n + 1)) ** 2
        solver = pps.FlexibleCG(grid, pps.ChebyshevIteration(11), tolerance=1e-10, max_iteration=20000,
                                form=case["form"], inner_tol=1e-5)
        solver.set_learned(net, k, gain, pps.LEARNED_PRECONDITIONER)
        solver.set_learned_cycle(5, 4, 8.0)
        s = {"net": net, "solver": solver, "b": _rhs(grid, seed)}
        s["x"] = torch.zeros_like(s["b"])
    elif kind == "batch":
        grids = [pps.BlockGrid.cube(m) for m in _batch_edges(case, seed)]
        inner = {"vcycle": 1e-5, "bicgstab": 3e-3}[case["method"]]
        batch = pps.Batch(grids, tolerance=1e-10, inner_tol=inner, method=case["method"])
        gen = _generator(seed)
        s = {"batch": batch, "x": []}
        for p, g in enumerate(grids):
            x, b = batch.field_device(p)
            s["x"].append(torch.as_tensor(_DeviceField(x, g.shape), device=DEV))
            torch.as_tensor(_DeviceField(b, g.shape), device=DEV)[g.unknowns()] = -_blobs(g.npglobal[0] - 2, gen)
    else:
        net = pps.UNet(CHANNELS, seed=1, linear=case["linear"])
        net.set_params(_initial_params(seed))
        x, t = _net_sample(case, seed)
        s = {"net": net, "shape": tuple(x.shape), "in": x, "target": t, "out": torch.zeros_like(x)}
    s["case"] = dict(case)
    torch.cuda.synchronize()   # the library's streams do not wait for torch's
    return s


# ---------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "operator":
        pps.apply_operator_noalloc(state["grid"], state["u"].data_ptr(), state["out"].data_ptr(),
                                   state["energy"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"out": state["out"], "energy": state["energy"]}
    if kind in ("solve", "learned"):
        x, b = state["x"], state["b"]
        if case.get("host"):
            x.fill(0.0)
            status = state["solver"](x, b)
        else:
            x.zero_()
            torch.cuda.current_stream().synchronize()   # the solver runs on its own stream
            status = state["solver"].solve_device(x.data_ptr(), b.data_ptr())
        return {"x": x, "status": status}
    if kind == "batch":
        torch._foreach_zero_(state["x"])
        torch.cuda.current_stream().synchronize()
        status = state["batch"].solve()
        return {"x": torch.cat([x.reshape(-1) for x in state["x"]]), "status": status}
    net, shape = state["net"], state["shape"]
    if kind == "forward":
        net.forward(shape, state["in"].data_ptr(), state["out"].data_ptr())
        return {"out": state["out"]}
    if kind == "gradients":
        loss, grads = net.gradients(shape, state["in"].data_ptr(), state["target"].data_ptr())
        return {"loss": loss, "grads": grads}
    loss = net.train_step(shape, state["in"].data_ptr(), state["target"].data_ptr(), case["lr"])
    return {"loss": loss, "params": net.get_params()}


# ---------------------------------------------------------------- what a pass cannot do without

def _conv_flops(case):
    v = case["nx"] * case["ny"] * case["nz"]
    per_level = (v, v, v / 8, v / 8, v / 64, v / 64, v / 8, v / 8, v, v, v)
    return sum(2.0 * 27 * cin * cout * n for (cin, cout), n in zip(LAYERS, per_level))


def work(case):
    """Bytes: the inputs read once and the outputs written once.  Operations: one
    application of the operator to the answer for a solve, the convolutions of the network."""
    kind = case["kind"]
    if kind in ("operator", "solve", "learned"):
        grid = _learned_grid(case) if kind == "learned" else _grid(case)
        n = grid.n_unknowns()
        return {"bytes": 16.0 * n, "flops": 10.0 * n}
    if kind == "batch":
        n = sum(m ** 3 for m in _batch_edges(case, 0))
        return {"bytes": 16.0 * n, "flops": 10.0 * n}
    v = case["nx"] * case["ny"] * case["nz"]
    params = sum(27 * cin * cout + cout for cin, cout in LAYERS)
    if kind == "forward":
        return {"bytes": 8.0 * v + 4.0 * params, "flops": _conv_flops(case)}
    first = 2.0 * 27 * v * LAYERS[0][1]   # no data gradient of the first layer
    moved = 8.0 * params if kind == "gradients" else 28.0 * params   # weights, gradients; Adam: p, m, v read and written
    return {"bytes": 8.0 * v + moved, "flops": 3.0 * _conv_flops(case) - first}


# ---------------------------------------------------------------- the same in 64 bits

def _axis_operator(n, h, neumann_upper):
    """Second difference on n unknowns, wall value 0 below; above, wall value 0 or a zero
    normal derivative (ghost value equal to the inner neighbour), made symmetric by the
    diagonal scaling that is returned with it."""
    t = np.diag(np.full(n, -2.0)) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)
    scale = np.ones(n)
    if neumann_upper:
        t[n - 1, n - 2] = t[n - 2, n - 1] = math.sqrt(2.0)
        scale[n - 1] = math.sqrt(0.5)
    return t / (h * h), scale


def _exact_solve(grid, b):
    """u with A u = b on the grid's unknowns, by the eigenvectors of the three axes."""
    shape = _unknown_shape(grid)
    u = b[grid.unknowns()].clone()
    vectors, values, scales = [], [], []
    for a, d in enumerate((2, 1, 0)):
        t, scale = _axis_operator(shape[a], grid.ds[d], grid.bcs[2 * d + 1] == 1)
        w, v = np.linalg.eigh(t)
        vectors.append(torch.from_numpy(v).to(DEV))
        values.append(torch.from_numpy(w).to(DEV))
        scales.append(torch.from_numpy(scale).to(DEV))
    scale = scales[0][:, None, None] * scales[1][None, :, None] * scales[2][None, None, :]
    u *= scale

    def along(t, mats):
        t = torch.matmul(t, mats[2])
        t = torch.matmul(mats[1].T, t)
        return torch.matmul(mats[0].T, t.reshape(t.shape[0], -1)).reshape(t.shape)

    u = along(u, vectors)
    u /= values[0][:, None, None] + values[1][None, :, None] + values[2][None, None, :]
    u = along(u, [v.T.contiguous() for v in vectors])
    u /= scale
    x = _padded(grid, u)
    inner = grid.unknowns()
    for a, d in enumerate((2, 1, 0)):   # the ghost layer above a Neumann face mirrors the inner neighbour
        if grid.bcs[2 * d + 1] == 1:
            ghost, mirror = list(inner), list(inner)
            ghost[a], mirror[a] = inner[a].stop, inner[a].stop - 2
            x[tuple(ghost)] = x[tuple(mirror)]
    return x


def _laplacian(grid, u):
    inner = tuple(slice(s.start, s.stop) for s in grid.unknowns())
    out = torch.zeros_like(u)
    for a, d in enumerate((2, 1, 0)):
        lo, hi = list(inner), list(inner)
        lo[a] = slice(inner[a].start - 1, inner[a].stop - 1)
        hi[a] = slice(inner[a].start + 1, inner[a].stop + 1)
        out[inner] += (u[tuple(lo)] - 2.0 * u[inner] + u[tuple(hi)]) / grid.ds[d] ** 2
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "operator":
        grid = _grid(case)
        u = _rhs(grid, seed)
        out = _laplacian(grid, u)
        return {"out": out, "energy": (u * out).sum().reshape(1)}
    if kind in ("solve", "learned"):
        grid = _learned_grid(case) if kind == "learned" else _grid(case)
        x = _exact_solve(grid, _rhs(grid, seed))
        return {"x": x.cpu().numpy() if case.get("host") else x, "status": None}
    if kind == "batch":
        gen = _generator(seed)
        parts = []
        for m in _batch_edges(case, seed):
            grid = pps.BlockGrid.cube(m)
            parts.append(_exact_solve(grid, _padded(grid, -_blobs(m, gen))).reshape(-1))
        return {"x": torch.cat(parts), "status": None}
    params = _initial_params(seed)
    weights = _unflatten(params, torch.float64)
    x, t = _net_sample(case, seed)
    x, t = x.double(), t.double()
    if kind == "forward":
        rms = torch.sqrt(torch.mean(x * x))
        with torch.no_grad():
            return {"out": _net_forward(weights, (x / rms)[None, None], case["linear"])[0, 0] * rms}
    loss = torch.mean((_net_forward(weights, x[None, None], case["linear"])[0, 0] - t) ** 2)
    loss.backward()
    g = _flatten([(w.grad, b.grad) for w, b in weights])
    if kind == "gradients":
        return {"loss": float(loss.detach()), "grads": g.cpu().numpy()}
    b1, b2, eps = ADAM
    g = g * min(1.0, 1.0 / float(torch.linalg.norm(g)))
    m, v = (1 - b1) * g, (1 - b2) * g * g
    p = torch.from_numpy(params).to(DEV, torch.float64)
    p = p - case["lr"] * (m / (1 - b1)) / (torch.sqrt(v / (1 - b2)) + eps)
    return {"loss": float(loss.detach()), "params": p.cpu().numpy()}
