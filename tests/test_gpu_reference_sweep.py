"""The dataflow form of the reference's natural-order Gauss-Seidel inside the
reference V-cycle (hpcgb200_problem_mg_ref) against the same V-cycle put
together from the launch-per-front sweep (hpcgb200_ref_symgs, itself bitwise
the reference's C loop): bit for bit at the edges of its ranges."""
import ctypes

import numpy as np
import pytest
import torch

import rochpcg_b200 as R
from gpu_util import dev_field, sync

pytestmark = pytest.mark.gpu


def _vp(v):
    return ctypes.c_void_p(v if isinstance(v, int) else v.data_ptr())


def _cycle(P, level, r):
    """src/ComputeMG_ref.cpp:37-62 with the launch-per-front sweeps."""
    s = _vp(P.stream_handle)
    d = P.dims[level]
    mat = [_vp(P.device_ptr(f, level)) for f in ("mtx_ind", "values", "nnz_in_row")]
    slot = _vp(P.device_ptr("diag_slot", level))
    x = torch.zeros_like(r)
    torch.cuda.synchronize()

    def smooth():
        assert P.L.hpcgb200_ref_symgs(*d, *mat, slot, _vp(r), _vp(x), s) == 0
        sync(P)

    smooth()
    if level + 1 < P.nlevels:
        y = torch.empty_like(r)
        torch.cuda.synchronize()
        assert P.L.hpcgb200_ref_spmv(*d, *mat, _vp(x), _vp(y), s) == 0
        f2c = dev_field(P, "f2c", level, np.int32).long()
        xc = _cycle(P, level + 1, (r[f2c] - y[f2c]).contiguous())
        x[f2c] += xc
        torch.cuda.synchronize()
        smooth()
    return x


def _compare(P, r):
    z = torch.full_like(r, 7.0)
    torch.cuda.synchronize()
    P.mg_ref(r.data_ptr(), z.data_ptr())
    sync(P)
    want = _cycle(P, 0, r)
    assert torch.equal(z.isnan(), want.isnan())
    assert torch.equal(z.nan_to_num(), want.nan_to_num())


def _normal(P, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(P.rows[0], dtype=torch.float64, device="cuda", generator=g)


# one group of planes and several, a last group that is not full, the largest
# line count of the dataflow form and the first one beyond it, long and short x
@pytest.mark.parametrize("dims", [(16, 16, 16), (104, 104, 104), (8, 40, 96), (184, 24, 16), (16, 256, 24),
                                  (16, 264, 24), (24, 152, 40), (40, 8, 184), (72, 64, 32)])
def test_reference_cycle_is_the_front_by_front_one(dims):
    with R.Problem(*dims, nlevels=3, keep_generated=True) as P:
        for seed in (1, 2):  # the second call reuses the workspace with another r
            _compare(P, _normal(P, seed))


def test_more_planes_than_a_grid_has_in_z():
    """Launch dimensions y and z end at 65535."""
    with R.Problem(4, 4, 65544, nlevels=1, keep_generated=True) as P:
        _compare(P, _normal(P, 5))


@pytest.mark.parametrize("level", [0, 1])
@pytest.mark.parametrize("slot", [0, 26])
def test_changed_matrix_takes_the_general_sweep(level, slot):
    """An off-diagonal that is not -1 (first and last slot of an interior row), set after a first call."""
    with R.Problem(32, 24, 40, nlevels=2, keep_generated=True) as P:
        r = _normal(P, 3)
        _compare(P, r)
        nx, ny, _ = P.dims[level]
        v = dev_field(P, "values", level, np.float64)
        v[((5 * ny + 4) * nx + 3) * 27 + slot] = -0.75
        torch.cuda.synchronize()
        _compare(P, r)


def test_nan_with_the_flag_bits_is_a_value():
    """A NaN input whose bits are the dataflow kernels' not-yet-computed pattern."""
    with R.Problem(24, 16, 160, nlevels=1, keep_generated=True) as P:
        r = _normal(P, 4)
        r.view(torch.int64)[P.rows[0] // 2] = -1
        _compare(P, r)
