"""The FP64 stencil V-cycle's one-row kernels on levels whose colour bricks are
not 4-aligned and which are too large for the one-cluster SymGS: the bits of the
FP64 ELL V-cycle, even and odd grids, blocks of rows full and ragged."""
import pytest
import torch

import rochpcg_b200 as R
from gpu_util import sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,nlevels", [((52, 52, 52), 1), ((100, 84, 68), 2), ((104, 104, 104), 2), ((66, 62, 34), 1),
                                          ((51, 43, 71), 1), ((130, 34, 46), 1), ((129, 65, 33), 1),
                                          # as many planes as a launch's z axis holds, and more
                                          ((4, 4, 131070), 1), ((4, 4, 131080), 1)])
def test_cycle_is_the_ell_one(dims, nlevels):
    with R.Problem(*dims, nlevels=nlevels) as P:
        assert P.stencil_ok(0)
        g = torch.Generator(device="cuda").manual_seed(sum(dims))
        r = torch.randn(P.rows[0], dtype=torch.float64, device="cuda", generator=g)
        z = [torch.empty_like(r) for _ in range(2)]
        torch.cuda.synchronize()
        P.mg(r.data_ptr(), z[0].data_ptr(), mode=R.MODE_FP64)
        P.mg(r.data_ptr(), z[1].data_ptr(), mode=R.MODE_FP64_STENCIL)
        sync(P)
        assert torch.equal(z[0], z[1])
        if nlevels == 1:
            P.symgs(0, r.data_ptr(), z[0].data_ptr())
            sync(P)
            assert torch.isfinite(z[0]).all()
