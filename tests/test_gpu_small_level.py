"""The one-cluster SymGS of small levels (csrc/small_level.cu) bit for bit
against the CPU restatement and against the launch-per-colour kernels, at the
edges of its shapes: one CTA and 2 to 16, full and ragged last plane pairs,
odd grids, the largest level it takes and the first it does not."""
import ctypes

import numpy as np
import pytest
import torch

import rochpcg_b200 as R
from gpu_util import dev_field, host, sync, to_dev
from oracle.oracle import ColoredProblem

pytestmark = pytest.mark.gpu

# rows of a pass per CTA at the limits: 640 threads (implicit), 512 (ELL values)
GRIDS = [(4, 4, 4), (8, 8, 8), (16, 16, 8), (16, 16, 10), (32, 4, 32), (4, 32, 34), (40, 32, 64), (40, 32, 66),
         (32, 32, 64), (34, 32, 64), (64, 40, 12), (20, 12, 62)]
ODD = [(5, 7, 9), (13, 13, 13), (25, 21, 17), (39, 31, 63), (4, 5, 35)]


def _mg(P, r, mode):
    z = torch.empty_like(r)
    torch.cuda.synchronize()
    P.mg(r.data_ptr(), z.data_ptr(), mode=mode)
    sync(P)
    return host(z)


@pytest.mark.parametrize("dims,nlevels", [(d, 2) for d in GRIDS] + [(d, 1) for d in ODD])
def test_cycle_bitwise(dims, nlevels):
    O = ColoredProblem(*dims, nlevels=nlevels)
    r = np.random.default_rng(sum(dims)).normal(size=O.levels[0].m)
    with R.Problem(*dims, nlevels=nlevels) as P:
        rd = to_dev(r)
        want = O.mg(r)
        assert np.array_equal(_mg(P, rd, R.MODE_FP64), want)
        assert np.array_equal(_mg(P, rd, R.MODE_FP64_STENCIL), want)
        assert np.array_equal(_mg(P, rd, R.MODE_MIXED), O.mg_f32(r.astype(np.float32)).astype(np.float64))


@pytest.mark.parametrize("dims", [(8, 8, 8), (24, 16, 20), (40, 32, 32), (13, 13, 13)])
@pytest.mark.parametrize("value", [-1.0, -0.75])
def test_full_step_with_any_values(dims, value):
    """The full step on the ELL values against the C ABI's launches, with the stencil's values and with one changed."""
    with R.Problem(*dims, nlevels=1) as P:
        m = P.rows[0]
        v = dev_field(P, "ell_val", 0, np.float64)
        v[3 * m + m // 2] = value
        g = torch.Generator(device="cuda").manual_seed(5)
        r = torch.randn(m, dtype=torch.float64, device="cuda", generator=g)
        x = torch.randn(m, dtype=torch.float64, device="cuda", generator=g)
        y, s = x.clone(), ctypes.c_void_p(P.stream_handle)
        torch.cuda.synchronize()
        vp = lambda t: ctypes.c_void_p(t if isinstance(t, int) else t.data_ptr())  # noqa: E731
        for _ in range(2):
            P.symgs(0, r.data_ptr(), x.data_ptr())
            sizes, offsets = P.field("sizes"), P.field("offsets")
            assert P.L.hpcgb200_symgs(m, 8, 6, sizes.ctypes.data_as(ctypes.c_void_p),
                                      offsets.ctypes.data_as(ctypes.c_void_p), vp(P.device_ptr("ell_col")),
                                      vp(P.device_ptr("ell_val")), vp(P.device_ptr("inv_diag")), vp(r), vp(y), s) == 0
        sync(P)
        assert torch.equal(x, y)
        P.symgs_zero(0, r.data_ptr(), x.data_ptr())
        assert P.L.hpcgb200_symgs_zero(m, 8, 6, sizes.ctypes.data_as(ctypes.c_void_p),
                                       offsets.ctypes.data_as(ctypes.c_void_p), vp(P.device_ptr("ell_col")),
                                       vp(P.device_ptr("ell_val")), vp(P.device_ptr("diag_idx")),
                                       vp(P.device_ptr("diag")), vp(P.device_ptr("inv_diag")), vp(r), vp(y), s) == 0
        sync(P)
        assert torch.equal(x, y)


def _vp(t):
    return ctypes.c_void_p(t if isinstance(t, int) else t.data_ptr())


def _launches(P, level, r, x, zero):
    """One SymGS step of a level by the C ABI's launch-per-colour kernels on its present ELL arrays."""
    sizes, offsets = P.field("sizes", level), P.field("offsets", level)
    lay = (P.rows[level], 8, 6, sizes.ctypes.data_as(ctypes.c_void_p), offsets.ctypes.data_as(ctypes.c_void_p))
    f = lambda *names: [_vp(P.device_ptr(n, level)) for n in names]  # noqa: E731
    s = ctypes.c_void_p(P.stream_handle)
    if zero:
        rc = P.L.hpcgb200_symgs_zero(*lay, *f("ell_col", "ell_val", "diag_idx", "diag", "inv_diag"), _vp(r), _vp(x), s)
    else:
        rc = P.L.hpcgb200_symgs(*lay, *f("ell_col", "ell_val", "inv_diag"), _vp(r), _vp(x), s)
    assert rc == 0


def _change(P, what):
    """Changes the level-0 ELL data of one row that has all its neighbours (and of one on a face)."""
    m = P.rows[0]
    col = dev_field(P, "ell_col", 0, np.int32).view(27, m)
    val = dev_field(P, "ell_val", 0, np.float64).view(27, m)
    inner = (col >= 0).all(0).nonzero().flatten()
    row = int(inner[len(inner) // 3]) if what != "diagonal" else int(inner[-1])  # one that is restricted
    face = int((col[26] < 0).nonzero().flatten()[0])
    if what == "column":  # the neighbouring row of the same colour
        col[4, row] += 1
    elif what == "last column of a face row":  # a slot that its faces leave empty
        col[26, face], val[26, face] = int(col[0, face]), -0.5
    elif what == "diagonal":
        val[int(dev_field(P, "diag_idx", 0, np.int32)[row]), row] = 30.0
    elif what == "diagonals' slot":
        dev_field(P, "diag_idx", 0, np.int32)[row] -= 1
    elif what == "injection":
        f = dev_field(P, "inj_f", 0, np.int32)
        f[:2] = f[:2].flip(0).clone()
    elif what == "value":
        val[7, row] = -0.25
    torch.cuda.synchronize()


CHANGES = ["none", "column", "last column of a face row", "diagonal", "diagonals' slot", "value", "injection"]


@pytest.mark.parametrize("dims", [(8, 8, 8), (16, 16, 16), (32, 24, 48)])
@pytest.mark.parametrize("what", CHANGES)
def test_cycle_on_changed_ell_arrays(dims, what):
    """The FP64 operators are those of the ELL arrays as they are, on small levels too."""
    with R.Problem(*dims, nlevels=2) as P:
        n, s = P.rows, ctypes.c_void_p(P.stream_handle)
        assert (dev_field(P, "inj_f", 0, np.int32).diff() == 1).all()  # what the one-cluster form counts on
        g = torch.Generator(device="cuda").manual_seed(8)
        r = torch.randn(n[0], dtype=torch.float64, device="cuda", generator=g)
        x = torch.randn(n[0], dtype=torch.float64, device="cuda", generator=g)
        _change(P, what)
        y = x.clone()
        torch.cuda.synchronize()
        P.symgs(0, r.data_ptr(), x.data_ptr())
        _launches(P, 0, r, y, False)
        sync(P)
        assert torch.equal(x, y)
        P.symgs_zero(0, r.data_ptr(), x.data_ptr())
        _launches(P, 0, r, y, True)
        sync(P)
        assert torch.equal(x, y)
        # the V-cycle (src/ComputeMG.cpp:72-101)
        rc, xc = (torch.zeros(n[1], dtype=torch.float64, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        f = lambda *names: [_vp(P.device_ptr(q)) for q in names]  # noqa: E731
        assert P.L.hpcgb200_restrict_fused(n[1], *f("inj_f", "inj_c"), n[0], *f("ell_col", "ell_val"), _vp(r), _vp(y),
                                           _vp(rc), s) == 0
        _launches(P, 1, rc, xc, True)
        sync(P)
        inj = dev_field(P, "inj_f", 0, np.int32).long()
        y[inj] += xc[dev_field(P, "inj_c", 0, np.int32).long()]
        torch.cuda.synchronize()
        _launches(P, 0, r, y, False)
        sync(P)
        assert np.array_equal(_mg(P, r, R.MODE_FP64), host(y))


def test_solve_on_changed_ell_arrays():
    """A captured FP64 solve and its V-cycle against the CPU restatement on the same changed arrays."""
    O = ColoredProblem(32, 32, 32)
    with R.Problem(32) as P:
        healthy = P.cg(8, 0.0)["hist"]
        for level, slot in ((0, 4), (1, 20)):
            lev = O.levels[level]
            row = int(np.flatnonzero((lev.ell_col >= 0).all(0))[11])
            lev.ell_val[slot, row] = -0.5
            lev.ell_col[4, row] += 1  # the neighbouring row of the same colour
            for f, a in (("ell_val", lev.ell_val), ("ell_col", lev.ell_col)):
                dev_field(P, f, level, a.dtype).copy_(torch.from_numpy(a.ravel()))
        torch.cuda.synchronize()
        r = np.random.default_rng(9).normal(size=O.levels[0].m)
        assert np.array_equal(_mg(P, to_dev(r), R.MODE_FP64), O.mg(r))
        got, want = P.cg(8, 0.0)["hist"], O.cg(8, 0.0)["hist"]
        # dot products in another order, as on the healthy matrix
        assert np.allclose(got, want, rtol=1e-8, atol=0) and not np.allclose(got, healthy, rtol=1e-6, atol=0)
