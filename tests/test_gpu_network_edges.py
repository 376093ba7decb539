"""The network's kernels (csrc/learned.cu) at the edges of their bricks and
rings: layer 1, layer 3 and layer 3's gradient on exact bricks, one point more
and less; the weight gradient for as many units as a CTA's two register buffers
and three stages can be caught with; the convolution's output on 16 and 32 byte
boundaries."""
import ctypes

import numpy as np
import pytest
import torch

import rochpcg_b200 as R
from oracle import oracle as O
from rochpcg_b200 import learned as LS

pytestmark = pytest.mark.gpu


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


def layers(w):
    return np.split(np.asarray(w), 3)


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("dims,nb", [((4, 8, 16), 2), ((5, 9, 17), 2), ((3, 7, 15), 3), ((1, 2, 3), 2), ((9, 1, 33), 1)])
def test_network_and_gradient(dims, nb, odd):
    rng = np.random.default_rng(sum(dims))
    per = int(np.prod(dims))
    w = LS.jacobi_weights(0.8, 0.15, 5)
    S = LS.Smoother(w, symmetry=LS.ODD if odd else LS.PLAIN)
    r = rng.standard_normal(nb * per).astype(np.float32)
    e = (rng.standard_normal(nb * per) * 0.05).astype(np.float32)
    rd, ed = torch.from_numpy(r).cuda(), torch.from_numpy(e).cuda()
    inv = LS.sample_norms(ed, dims, nb, 0)
    y = S.forward(rd, dims, nb)
    loss, dw = S.loss_grad(rd, ed, inv, dims, nb, 1.0, 0)
    torch.cuda.synchronize()
    w1, w2, w3 = layers(w)
    want = np.zeros(3 * 27 * 256)
    for b in range(nb):
        sl = slice(b * per, (b + 1) * per)
        z = O.net_forward(dims, w1, w2, w3, r[sl])[0]
        if odd:
            z = 0.5 * (z - O.net_forward(dims, w1, w2, w3, -r[sl])[0])
        # BF16 activations that a summation order rounds the other way: 2^-8 of one of 432 terms
        assert np.max(np.abs(y.cpu().numpy()[sl] - z)) <= 2e-3 * np.max(np.abs(z))
        want += np.concatenate(O.net_loss_grad(dims, w1, w2, w3, r[sl], e[sl], odd=odd)[1])
    for a, b in zip(layers(dw.cpu().numpy()), layers(want)):
        assert np.linalg.norm(a - b) <= 3e-3 * np.linalg.norm(b)


@pytest.mark.parametrize("dims,nb", [((8, 3, 16), k) for k in (1, 2, 148, 149, 296, 297, 445, 600)] + [((9, 4, 17), 37)])
def test_weight_gradient_units(dims, nb):
    """Small whole numbers: every partial sum is exact in FP32, and so are the results."""
    L = R.load()
    nz, ny, nx = dims
    g = torch.Generator(device="cuda").manual_seed(nb)
    x = torch.randint(-2, 3, (nb, nz, ny, nx, 16), device="cuda", generator=g).to(torch.bfloat16)
    d = torch.randint(-2, 3, (nb, nz, ny, nx, 16), device="cuda", generator=g).to(torch.bfloat16)
    partial = torch.empty(L.hpcgb200_conv_wgrad_partial_bytes(nb, nz, ny, nx) // 4, device="cuda")
    dw = torch.empty(27, 16, 16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.hpcgb200_conv16_wgrad(nb, nz, ny, nx, vp(x), vp(d), vp(partial), vp(dw), vp(status), stream) == 0
    torch.cuda.synchronize()
    assert status.item() == 0
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    for t in range(27):
        a, b, c = t // 9, t // 3 % 3, t % 3
        want = torch.einsum("nzyxi,nzyxo->io", xp[:, a:a + nz, b:b + ny, c:c + nx], d.double())
        assert torch.equal(dw[t].double(), want)


@pytest.mark.parametrize("mode", [0, 1])
def test_convolution_output_alignment(mode):
    L = R.load()
    nb, nz, ny, nx = 2, 5, 9, 17
    n = nb * nz * ny * nx
    g = torch.Generator(device="cuda").manual_seed(3)
    x, act = (torch.randn(n * 16, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    w = torch.randn(27 * 256, device="cuda", generator=g)
    wB = torch.empty(L.hpcgb200_conv_weight_tile_bytes(), dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.hpcgb200_conv_prepare_weights(vp(w), vp(wB), 0, stream) == 0
    got = []
    for shift in (0, 8):  # elements: 0 and 16 bytes
        out = torch.full((n * 16 + 16,), 7.0, dtype=torch.bfloat16, device="cuda")
        assert out.data_ptr() % 32 == 0
        o = out[shift:shift + n * 16]
        assert L.hpcgb200_conv16(nb, nz, ny, nx, vp(x), vp(wB), mode, vp(o), vp(act), vp(status), stream) == 0
        torch.cuda.synchronize()
        assert torch.all(out[:shift] == 7) and torch.all(out[shift + n * 16:] == 7)
        got.append(o.clone())
    assert status.item() == 0 and torch.equal(got[0], got[1])
