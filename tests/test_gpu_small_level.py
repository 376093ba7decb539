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
