"""A problem's device memory: everything goes back to the driver when it is
closed (its arrays come from chunks that nothing may keep), also after a set-up
that fails, and problems alive together do not share arrays."""
import pytest
import torch

import rochpcg_b200 as R
from gpu_util import dev_field

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("dims,keep", [((16, 16, 16), False), ((40, 48, 56), True), ((104, 104, 104), False),
                                       ((168, 168, 168), True)])
def test_memory_returns(dims, keep):
    with R.Problem(*dims, keep_generated=keep) as P:  # the runtime's own buffers
        P.cg(2, 0.0)
    before = _free()
    for _ in range(2):
        with R.Problem(*dims, keep_generated=keep) as P:
            P.cg(2, 0.0, mode=R.MODE_MIXED)
            if keep:
                P.cg_ref(1, 0.0)
    assert _free() == before


def test_failed_setup_returns_its_memory():
    def fail():
        with pytest.raises(R.HpcgError):
            R.Problem(32, 24, 16)  # the colouring of its 4 x 3 x 2 level does not end

    fail()
    before = _free()
    fail()
    assert _free() == before


def test_live_problems_are_apart():
    Ps = [R.Problem(32), R.Problem(40, 32, 48), R.Problem(32)]
    spans = []
    for P in Ps:
        for level in range(4):
            for f, kind in (("perm", "i4"), ("ell_col", "i4"), ("ell_val", "f8"), ("diag", "f8"), ("inv_diag", "f8"),
                            ("diag32", "f4"), ("colors", "i4")):
                t = dev_field(P, f, level, kind)
                assert t.data_ptr() % 256 == 0
                spans.append((t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()))
    spans.sort()
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    want = Ps[0].cg(20, 0.0)["hist"]
    Ps[1].close()
    assert (Ps[2].cg(20, 0.0)["hist"] == want).all()
    for P in Ps:
        P.close()
