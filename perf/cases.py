"""Workloads this framework is timed on, through its public Python entry points.

Three families: multigrid cycles and CG solves of the HPCG problem in every
solver mode (a Problem handle the program keeps, new right-hand sides), the
benchmark protocol's natural-order reference V-cycle, and the learned
smoother's training gradient and evaluation.  Sizes run from the reference's
smallest local grid (16 points an axis) to 320^3, the mixed-precision headline
grid; drawn cases also take uneven axes and odd coarse levels.

`exact` restates each path in 64 bits with plain torch: the multicolour
V-cycle on parity classes, the conjugate-gradient recurrence, the sequential
natural-order Gauss-Seidel, and the three-layer convolution with its gradient.
"""
import math

import numpy as np
import torch

import rochpcg_b200 as R
from rochpcg_b200 import learned as LN

MODES = {"fp64": R.MODE_FP64, "stencil": R.MODE_FP64_STENCIL, "mixed": R.MODE_MIXED, "learned": R.MODE_LEARNED}
LEVELS = 4
TOL = 1e-9
MAX_ITER = 1000


def _grid(kind, mode, nx, ny, nz, **more):
    return dict(kind=kind, mode=mode, nx=nx, ny=ny, nz=nz, **more)


def listed():
    return [
        # the smallest local grid of the reference's tests: one V-cycle through the operator API, all launch latency
        dict(_grid("mg", "fp64", 16, 16, 16), name="mg_fp64_16"),
        # HPCG's default local grid (104^3): coarse levels of 52, 26 and 13 points, the last one odd
        dict(_grid("mg", "mixed", 104, 104, 104), name="mg_mixed_104"),
        # an uneven grid in FP64 without matrix reads, one V-cycle
        dict(_grid("mg", "stencil", 192, 96, 160), name="mg_stencil_192x96x160"),
        # one timed CG set of the HPCG protocol: fixed iterations, general FP64 matrix, the benchmark's 256^3 grid
        dict(_grid("cg", "fp64", 256, 256, 256, iters=50), name="cg_fp64_256"),
        # the same set on an uneven grid with the implicit FP64 operator
        dict(_grid("cg", "stencil", 200, 168, 136, iters=50), name="cg_stencil_200x168x136"),
        # the mixed-precision headline: a solve of a new right-hand side to 1e-9 on 320^3
        dict(_grid("cg", "mixed", 320, 320, 320, iters=0), name="cg_mixed_320"),
        # the learned smoother's headline grid, to 1e-9
        dict(_grid("cg", "learned", 256, 256, 256, iters=0), name="cg_learned_256"),
        # a small solve end to end from host memory: copies in, solve, copy out
        dict(_grid("host", "mixed", 64, 64, 64), name="host_mixed_64"),
        # the command-line solver's whole run: generate, optimize, solve, fetch x
        dict(_grid("oneshot", "fp64", 128, 128, 128), name="oneshot_fp64_128"),
        # the protocol's reference phase: one natural-order V-cycle on the default local grid
        dict(_grid("mgref", "fp64", 104, 104, 104), name="mgref_104"),
        # one training batch of the smoother: 64 level-2 samples of a 64^3 grid
        dict(_grid("train", "odd", 16, 16, 16, nb=64), name="train_64x16"),
        # the network applied to one large level
        dict(_grid("net", "odd", 128, 128, 128, nb=1), name="net_128"),
    ]


def _axis(rng, lo, hi, step):
    """A multiple of step in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, step * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)))


def _axes(rng, lo, hi, step, most):
    while True:
        d = [_axis(rng, lo, hi, step) for _ in range(3)]
        if d[0] * d[1] * d[2] <= most:
            return d


def draw(rng):
    kind, mode = rng.choice([("mg", "fp64"), ("mg", "stencil"), ("mg", "mixed"), ("cg", "fp64"), ("cg", "stencil"),
                             ("cg", "mixed"), ("cg", "learned"), ("host", "mixed"), ("host", "stencil"),
                             ("oneshot", "fp64"), ("oneshot", "mixed"), ("mgref", "fp64"), ("train", "odd"),
                             ("net", "odd")])
    if kind == "train":
        n = [_axis(rng, 6, 34, 1) for _ in range(3)]
        most = max(1, 262144 // (n[0] * n[1] * n[2]))
        return _grid(kind, mode, *n, nb=rng.randint(1, min(64, most)))
    if kind == "net":
        return _grid(kind, mode, *_axes(rng, 9, 144, 1, 128 ** 3), nb=rng.randint(1, 2))
    if mode == "learned":
        return _grid(kind, mode, *_axes(rng, 64, 256, 32, 192 ** 3), iters=0)
    if kind == "cg":
        return _grid(kind, mode, *_axes(rng, 32, 256, 8, 192 ** 3), iters=rng.choice([0, 25, 50]))
    if kind in ("mgref", "oneshot"):
        return _grid(kind, mode, *_axes(rng, 32, 128, 8, 128 ** 3))
    # the largest grid of the listed V-cycles and host solves, and down to the smallest
    return _grid(kind, mode, *_axes(rng, 32, 256, 8, 224 ** 3))


# ------------------------------------------------------------------ inputs


def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 2654435761 + salt) % (1 << 62))


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _normal(case, seed):
    """N(0,1) right-hand side in natural order, on the device, shape (nz, ny, nx)."""
    nx, ny, nz = _dims(case)
    return torch.randn(nz, ny, nx, dtype=torch.float64, device="cuda", generator=_gen(seed, 1))


def _samples(case, seed):
    """Training pairs: e a random field damped towards smoothness, r = A e (the stencil), as the V-cycle hands them
    down; both FP32."""
    nx, ny, nz = _dims(case)
    e = torch.randn(case["nb"], nz, ny, nx, dtype=torch.float64, device="cuda", generator=_gen(seed, 2))
    e = 0.3 * e + _box(e) / 27.0
    e = (0.05 * e).float().contiguous()
    d = e.double()
    return (27.0 * d - _box(d)).float().contiguous(), e


class _View:
    """A problem's device array for torch (CUDA array interface, no copy): the tensor keeps the problem alive."""

    def __init__(self, P, field, kind):
        self.owner = P
        self.__cuda_array_interface__ = {"shape": (P.rows[0],), "typestr": kind, "data": (P.device_ptr(field), False),
                                         "version": 3}


def prepare(case, seed):
    kind, mode = case["kind"], case["mode"]
    s = dict(case=case)
    if kind in ("train", "net"):
        s["net"] = LN.Smoother.load()
        s["r"], s["e"] = _samples(case, seed)
        nx, ny, nz = _dims(case)
        if kind == "train":
            s["inv"] = LN.sample_norms(s["e"], (nz, ny, nx), case["nb"], kind=1)
        torch.cuda.synchronize()
        return s
    b = _normal(case, seed)
    if kind == "oneshot":
        s["b"] = b.reshape(-1).cpu().numpy()
        return s
    P = s["P"] = R.Problem(*_dims(case), nlevels=LEVELS, keep_generated=kind == "mgref")
    s["stream"] = torch.cuda.ExternalStream(P.stream_handle)
    if mode == "learned":
        P.set_smoother(LN.Smoother.load())
    if kind == "mg":
        perm = torch.as_tensor(_View(P, "perm", "<i4"), device="cuda")
        s["r"] = torch.empty(P.rows[0], dtype=torch.float64, device="cuda")
        s["r"][perm.long()] = b.reshape(-1)
        s["z"] = torch.empty_like(s["r"])
    elif kind == "mgref":
        s["r"] = b.reshape(-1).contiguous()
        s["z"] = torch.empty_like(s["r"])
    elif kind == "cg":
        P.set_rhs(b.reshape(-1).cpu().numpy())
        s["x"] = torch.as_tensor(_View(P, "x", "<f8"), device="cuda")
        s["x"].owner = P
    else:
        s["b"] = b.reshape(-1).cpu().pin_memory()
        s["x"] = torch.empty(P.rows[0], dtype=torch.float64).pin_memory()
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind, mode = case["kind"], case["mode"]
    if kind == "train":
        loss, dw = s["net"].loss_grad(s["r"], s["e"], s["inv"], _dims(case)[::-1], nb=case["nb"],
                                      scale=1.0 / case["nb"], kind=1)
        return dict(loss=loss, dw=dw)
    if kind == "net":
        return s["net"].forward(s["r"], _dims(case)[::-1], nb=case["nb"])
    if kind == "oneshot":
        with R.Problem(*_dims(case), nlevels=LEVELS) as P:
            P.set_rhs(s["b"])
            P.cg(MAX_ITER, TOL, mode=MODES[mode])
            return P.get_x()
    P = s["P"]
    if kind == "host":
        P.solve_host(s["b"], s["x"], MAX_ITER, TOL, mode=MODES[mode])
        return s["x"]
    if kind == "cg":
        if case["iters"]:
            h = P.cg(case["iters"], 0.0, mode=MODES[mode])
            return dict(x=s["x"], hist=h["hist"])
        P.cg(MAX_ITER, TOL, mode=MODES[mode])
        return s["x"]
    # the handle's operators run on its own stream
    s["stream"].wait_stream(torch.cuda.current_stream())
    if kind == "mgref":
        P.mg_ref(s["r"].data_ptr(), s["z"].data_ptr())
    else:
        P.mg(s["r"].data_ptr(), s["z"].data_ptr(), mode=MODES[mode])
    torch.cuda.current_stream().wait_stream(s["stream"])
    return s["z"]


# -------------------------------------------------------------------- work


def _levels(case):
    return [tuple(v >> l for v in _dims(case)) for l in range(LEVELS)]


def _nnz(d):
    return math.prod(3 * v - 2 for v in d)


def work(case):
    """Bytes and operations one pass cannot do without.  A V-cycle or CG iteration reads every level's operator once
    (12 B a nonzero slot of the general matrix, the diagonal alone where the stencil is implicit) and its vectors
    once; a solve to 1e-9 takes about 0.6 n iterations on an n^3 grid."""
    kind, mode = case["kind"], case["mode"]
    m = math.prod(_dims(case))
    if kind in ("train", "net"):
        pts = m * case["nb"]
        fwd = 2 * 2 * 27 * (16 + 256 + 16) * pts  # both branches of the odd evaluation
        if kind == "net":
            return dict(bytes=8 * pts, flops=fwd)
        return dict(bytes=8 * pts + 4 * LN.WEIGHTS, flops=3 * fwd)
    lv = _levels(case)
    rows = [math.prod(d) for d in lv]
    if mode == "fp64":
        op = sum(12 * 27 * r for r in rows)
        op0 = 0
    elif mode == "stencil":
        op = sum(8 * r for r in rows)
        op0 = 8 * rows[0]
    else:
        op = sum(4 * r for r in rows)
        op0 = 8 * rows[0]
    cyc = sum(10 * _nnz(d) for d in lv[:-1]) + 4 * _nnz(lv[-1])
    if kind in ("mg", "mgref"):
        return dict(bytes=op + 16 * m, flops=cyc)
    n = case.get("iters") or round(0.6 * m ** (1 / 3))
    by, fl = n * (op + op0 + 48 * m), n * (cyc + 2 * _nnz(lv[0]) + 12 * m)
    if kind == "oneshot":
        by += sum(12 * 27 * r for r in rows) + 16 * m
    elif kind == "host":
        by += 16 * m
    return dict(bytes=by, flops=fl)


def tolerance(case):
    """About four times what the path differs from `exact` by: FP64 rounding, the FP32 V-cycle's rounding, the stopping
    error of a solve to 1e-9, BF16 activations."""
    kind, mode = case["kind"], case["mode"]
    if kind == "train":
        return dict(rel=3e-2)
    if kind == "net":
        return dict(rel=1.7e-2)
    if kind in ("mg", "mgref"):
        return dict(rel=6e-7) if mode == "mixed" else dict(rel=2e-15)
    if kind == "cg" and case["iters"] and mode != "mixed":
        return dict(rel=1e-12)
    return dict(rel=5e-7)


# ---------------------------------------------------- 64-bit restatements


def _box(x):
    """Sum over the 27-point box around every point (zero outside), last three axes."""
    for d in (-1, -2, -3):
        n = x.shape[d]
        y = x.clone()
        if n > 1:
            y.narrow(d, 1, n - 1).add_(x.narrow(d, 0, n - 1))
            y.narrow(d, 0, n - 1).add_(x.narrow(d, 1, n - 1))
        x = y
    return x


def _apply(x):
    return 27.0 * x - _box(x)


# colour of each parity class (4 px + 2 py + pz) of the grid's points, in sweep order
_CLASS_OF_COLOUR = [7, 6, 1, 2, 5, 4, 3, 0]


class _Cycle:
    """The multicolour V-cycle: zero-guess symmetric sweep, injected residual, coarse solve, correction, sweep."""

    def __init__(self, dims):
        self.dims = dims

    @staticmethod
    def _update(xp, r, cls):
        px, py, pz = (cls >> 2) & 1, (cls >> 1) & 1, cls & 1
        nz, ny, nx = r.shape
        bz, by, bx = (nz - pz + 1) // 2, (ny - py + 1) // 2, (nx - px + 1) // 2
        a = sum(xp[pz + d:pz + d + 2 * bz - 1:2] for d in range(3))
        a = sum(a[:, py + d:py + d + 2 * by - 1:2] for d in range(3))
        a = sum(a[:, :, px + d:px + d + 2 * bx - 1:2] for d in range(3))
        own = xp[1 + pz::2, 1 + py::2, 1 + px::2][:bz, :by, :bx]
        own.copy_((r[pz::2, py::2, px::2] + (a - own)) / 26.0)

    def sweep(self, xp, r):
        for c in list(range(8)) + list(range(6, -1, -1)):
            self._update(xp, r, _CLASS_OF_COLOUR[c])

    def __call__(self, r, level=0):
        nx, ny, nz = (v >> level for v in self.dims)
        xp = torch.zeros(nz + 2, ny + 2, nx + 2, dtype=torch.float64, device=r.device)
        x = xp[1:-1, 1:-1, 1:-1]
        self.sweep(xp, r)
        if level + 1 < LEVELS:
            res = (r - _apply(x))[::2, ::2, ::2].contiguous()
            x[::2, ::2, ::2] += self(res, level + 1)
            self.sweep(xp, r)
        return x.contiguous()


class _NaturalCycle:
    """The reference V-cycle: sequential Gauss-Seidel in natural order, run front by front."""

    def __init__(self, dims, device):
        self.dims, self.fronts = dims, []
        for l in range(LEVELS):
            nx, ny, nz = (v >> l for v in dims)
            iz, iy, ix = torch.meshgrid(torch.arange(nz), torch.arange(ny), torch.arange(nx), indexing="ij")
            t = (ix + 2 * iy + 4 * iz).reshape(-1).to(device)
            at = (((iz + 1) * (ny + 2) + iy + 1) * (nx + 2) + ix + 1).reshape(-1).to(device)
            order = torch.argsort(t, stable=True)
            counts = torch.bincount(t).tolist()
            self.fronts.append((order, at[order], [c for c in counts if c]))
        self.device = device

    def sweep(self, xp, r, level):
        nx, ny, _ = (v >> level for v in self.dims)
        order, at, counts = self.fronts[level]
        off = torch.tensor([(a * (ny + 2) + b) * (nx + 2) + c for a in (-1, 0, 1) for b in (-1, 0, 1)
                            for c in (-1, 0, 1)], device=self.device)
        xf, rs = xp.reshape(-1), r.reshape(-1)[order]
        starts = np.concatenate([[0], np.cumsum(counts)])
        for k in list(range(len(counts))) + list(range(len(counts) - 1, -1, -1)):
            lo, hi = int(starts[k]), int(starts[k + 1])
            i = at[lo:hi]
            xf[i] = (rs[lo:hi] + xf[i[:, None] + off].sum(1) - xf[i]) / 26.0

    def __call__(self, r, level=0):
        nx, ny, nz = (v >> level for v in self.dims)
        xp = torch.zeros(nz + 2, ny + 2, nx + 2, dtype=torch.float64, device=r.device)
        x = xp[1:-1, 1:-1, 1:-1]
        self.sweep(xp, r, level)
        if level + 1 < LEVELS:
            res = (r - _apply(x))[::2, ::2, ::2].contiguous()
            x[::2, ::2, ::2] += self(res, level + 1)
            self.sweep(xp, r, level)
        return x.contiguous()


def _pcg(b, cycle, iters, tol):
    x = torch.zeros_like(b)
    r = b.clone()
    hist = [float(r.norm())]
    p, old = None, 1.0
    for _ in range(iters):
        if hist[-1] <= tol * hist[0]:
            break
        z = cycle(r)
        rz = float((r * z).sum())
        p = z if p is None else z + (rz / old) * p
        old = rz
        q = _apply(p)
        alpha = rz / float((p * q).sum())
        x += alpha * p
        r -= alpha * q
        hist.append(float(r.norm()))
    return x, hist


def _permuted(x, case):
    """Natural order (nz, ny, nx) -> the colour order: the eight parity classes in sweep order, each in natural
    order."""
    out = []
    for cls in _CLASS_OF_COLOUR:
        out.append(x[cls & 1::2, (cls >> 1) & 1::2, (cls >> 2) & 1::2].reshape(-1))
    return torch.cat(out)


def _taps(x):
    """The 27 shifted copies of (n, nz, ny, nx, c), zero outside, in (dz, dy, dx) order."""
    nz, ny, nx = x.shape[1:4]
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    for a in range(3):
        for b in range(3):
            for c in range(3):
                yield p[:, a:a + nz, b:b + ny, c:c + nx]


def _conv(x, w):
    return sum(t @ w[k] for k, t in enumerate(_taps(x)))


def _network(r, w):
    a = torch.relu(_conv(r[..., None], w[0][:, :1, :]))
    a = torch.relu(_conv(a, w[1]))
    return _conv(a, w[2][:, :, :1])[..., 0]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "net"):
        w = torch.from_numpy(LN.read_weights()[0]).cuda().double().reshape(3, 27, 16, 16)
        r, e = (v.double() for v in _samples(case, seed))
        if kind == "net":
            return 0.5 * (_network(r, w) - _network(-r, w)).reshape(-1)
        w.requires_grad_(True)
        d = 0.5 * (_network(r, w) - _network(-r, w)) - e
        sums = ((d * _apply(d)).sum((1, 2, 3)) / (e * _apply(e)).sum((1, 2, 3)))
        loss = sums.sum() / case["nb"]
        loss.backward()
        return dict(loss=float(loss), dw=w.grad.reshape(-1))
    b = _normal(case, seed)
    if kind == "mgref":
        return _NaturalCycle(_dims(case), b.device)(b).reshape(-1)
    cycle = _Cycle(_dims(case))
    if kind == "mg":
        return _permuted(cycle(b), case)
    if kind == "cg" and case["iters"]:
        x, hist = _pcg(b, cycle, case["iters"], 0.0)
        return dict(x=_permuted(x, case), hist=np.array(hist))
    if kind == "cg" and b.numel() > 300 ** 3:
        x, _ = _pcg(b, cycle, MAX_ITER, 1e-11)
        return _permuted(x, case)
    x, _ = _pcg(b, cycle, MAX_ITER, 1e-13)
    if kind == "cg":
        return _permuted(x, case)
    x = x.reshape(-1)
    return x.cpu().numpy()
