"""CPU restatement of the tcgen05 network kernels' issue plans and data
layouts (rochpcg_b200/csrc/learned.cu).  k_conv16: the weight slot order, the
MMAs per (staged plane, row shift) with the dz and dx taps stacked in N, their
accumulate flags, the shared-memory and TMEM ranges they touch, and the
epilogue's combination of the dx blocks of neighbouring rows -- checked
exhaustively for brick depths 1-5 and numerically against a direct 3x3x3
convolution of one brick.  k_layer3_tc: the same plan with one output channel
and the odd pair folded into K.  k_layer1_tc: the shifted runs and the product.
k_conv16_wgrad: one unit's MMAs and the sums over its lines."""
import numpy as np
import pytest

KTX, KTY = 16, 8          # staged x width (14 outputs + halo), output y
KHY = KTY + 2
CH = 16
PLANE_COLS = 3 * CH       # TMEM columns of one output plane: 3 dx blocks x 16 channels
TILE = CH * CH * 2        # bytes of one tap's 16 x 16 BF16 weight tile
TMEM_COLS = 512


def weight_slot(t):
    """Tile slot of tap t = (dz+1)*9 + (dy+1)*3 + (dx+1): [dy][dz = +1, 0, -1][dx]."""
    return ((t // 3) % 3) * 9 + (2 - t // 9) * 3 + t % 3


def plan(ktz):
    """(plane q, row shift dyi, first output plane, last output plane, accumulate)."""
    for q in range(ktz + 2):
        lo, hi = max(q - 2, 0), min(q, ktz - 1)
        for dyi in range(3):
            if q <= ktz - 1 and dyi == 0:
                if hi > lo:
                    yield q, dyi, lo, hi - 1, 1
                yield q, dyi, hi, hi, 0
            else:
                yield q, dyi, lo, hi, 1


def test_weight_slots_are_a_permutation_in_dy_dz_dx_order():
    slots = [weight_slot(t) for t in range(27)]
    assert sorted(slots) == list(range(27))
    for t in range(27):
        dz, dy, dx = t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1
        assert weight_slot(t) == (dy + 1) * 9 + (1 - dz) * 3 + (dx + 1)


@pytest.mark.parametrize("ktz", [1, 2, 3, 4, 5])
def test_plan_covers_every_tap_once(ktz):
    touched, cover, n = set(), set(), 0
    for q, dyi, m0, m1, acc in plan(ktz):
        n += 1
        N = (m1 - m0 + 1) * PLANE_COLS
        assert N % 16 == 0 and 16 <= N <= 256                         # kind::f16 with M = 128
        b_off = dyi * 9 * TILE + (m0 - q + 2) * 3 * TILE
        assert 0 <= b_off and b_off + N * 2 * CH <= 27 * TILE          # inside the weight tiles
        assert (q * KHY + dyi) * KTX + 128 <= KTX * KHY * (ktz + 2)   # A rows inside the staged box
        for a in (0, 1):                                               # both accumulators
            assert a * ktz * PLANE_COLS + (m1 + 1) * PLANE_COLS <= TMEM_COLS
        for mt in range(m0, m1 + 1):
            dz = 1 - (mt - q + 2)
            assert dz in (-1, 0, 1) and q == mt + 1 + dz
            assert (mt in touched) == (acc == 1)                       # first write clears, later ones add
            touched.add(mt)
            for dx in (-1, 0, 1):
                key = (mt, dz, dyi - 1, dx)
                assert key not in cover
                cover.add(key)
    assert len(cover) == 27 * ktz
    assert n == 3 * (ktz + 2) + ktz - 1                                # 21 for ktz = 4


@pytest.mark.parametrize("ktz", [1, 4])
def test_plan_and_epilogue_equal_a_direct_convolution(ktz):
    rng = np.random.default_rng(ktz)
    box = rng.standard_normal((ktz + 2, KHY, KTX, CH))                 # staged [z][y][x][ci], halo included
    w = rng.standard_normal((27, CH, CH))                              # w[tap][ci][co]
    # B operand rows: slot * 16 + co, K = ci
    B = np.zeros((27 * CH, CH))
    for t in range(27):
        B[weight_slot(t) * CH:(weight_slot(t) + 1) * CH, :] = w[t].T
    D = np.zeros((128, ktz * PLANE_COLS))
    for q, dyi, m0, m1, acc in plan(ktz):
        A = box[q, dyi:dyi + KTY, :, :].reshape(128, CH)               # row m = y * 16 + x of the shifted plane
        r0 = (dyi * 9 + (m0 - q + 2) * 3) * CH
        nrows = (m1 - m0 + 1) * PLANE_COLS
        prod = A @ B[r0:r0 + nrows].T
        cols = slice(m0 * PLANE_COLS, m0 * PLANE_COLS + nrows)
        D[:, cols] = prod if acc == 0 else D[:, cols] + prod
    for mt in range(ktz):
        blk = D[:, mt * PLANE_COLS:(mt + 1) * PLANE_COLS].reshape(KTY, KTX, 3, CH)
        # out(x) = D_{dx=-1}[x - 1] + D_{dx=0}[x] + D_{dx=+1}[x + 1] for the 14 inner columns
        got = blk[:, 0:14, 0] + blk[:, 1:15, 1] + blk[:, 2:16, 2]
        want = np.zeros((KTY, 14, CH))
        for t in range(27):
            dz, dy, dx = t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1
            src = box[mt + 1 + dz, 1 + dy:1 + dy + KTY, 1 + dx:1 + dx + 14, :]
            want += src @ w[t]
        assert np.allclose(got, want, rtol=1e-12, atol=1e-12)


# ---- layer 3 (k_layer3_tc): the same plan with one output channel

P3 = 16  # columns of one output plane: three dx taps, the others zero


def test_layer3_plan_and_pair_folding_equal_the_odd_conv():
    """Weight tile (dy, dz) has its three dx taps in columns 0-2; the second
    branch multiplies the negated weights, both halved, into the same
    accumulator, which then holds (conv(a+) - conv(a-)) / 2."""
    rng = np.random.default_rng(3)
    ktz = 4
    pos, neg = rng.standard_normal((2, ktz + 2, KHY, KTX, CH))
    w = rng.standard_normal((27, CH))                                  # w3[t][ci][0]
    B = np.zeros((9 * P3, CH))                                         # rows (dy, dz = +1, 0, -1, column)
    for tile in range(9):
        for col in range(3):
            B[tile * P3 + col] = 0.5 * w[(2 - tile % 3) * 9 + tile // 3 * 3 + col]
    D = np.full((128, ktz * P3), np.nan)
    n = 0
    for q, dyi, m0, m1, acc in plan(ktz):
        r0 = (dyi * 3 + m0 - q + 2) * P3
        nrows = (m1 - m0 + 1) * P3
        assert nrows in (16, 32, 48) and 0 <= r0 and r0 + nrows <= B.shape[0]
        cols = slice(m0 * P3, m0 * P3 + nrows)
        for box, sign, add in ((pos, 1.0, acc), (neg, -1.0, 1)):
            prod = box[q, dyi:dyi + KTY].reshape(128, CH) @ (sign * B[r0:r0 + nrows]).T
            D[:, cols] = prod if add == 0 else D[:, cols] + prod
            n += 1
    assert n == 42 and 2 * ktz * P3 <= 128                             # two accumulators in 128 columns
    for mt in range(ktz):
        blk = D[:, mt * P3:(mt + 1) * P3].reshape(KTY, KTX, P3)
        got = blk[:, 0:14, 0] + blk[:, 1:15, 1] + blk[:, 2:16, 2]
        want = np.zeros((KTY, 14))
        for t in range(27):
            dz, dy, dx = t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1
            sl = (mt + 1 + dz, slice(1 + dy, 1 + dy + KTY), slice(1 + dx, 15 + dx))
            want += 0.5 * (pos[sl] - neg[sl]) @ w[t]
        assert np.allclose(got, want, rtol=1e-12, atol=1e-12)
        assert not blk[..., 3:].any()


# ---- layer 1 (k_layer1_tc): taps as K, the operand MN-major

K1_GROUP, K1_PLANE = 32 * 16 + 16, 16 * (32 * 16 + 16)  # bytes of an 8-point group and of a plane


def k1_off(r, c8):
    """Byte offset of weight row r, 8-element K chunk c8."""
    return (r >> 3) * 512 + c8 * 128 + (r & 7) * 16


def test_layer1_weight_operand():
    """The MMA's K halves start 256 B apart with LBO 128 and SBO 512; 16 rows x 32 taps end at 1 KB."""
    for r in range(16):
        for c in range(4):
            kh, cc = divmod(c, 2)
            assert k1_off(r, c) == kh * 256 + (r >> 3) * 512 + cc * 128 + (r & 7) * 16
    assert max(k1_off(co, t >> 3) + (t & 7) * 2 for co in range(16) for t in range(32)) == 1022


def test_layer1_runs_make_the_operand_of_the_conv():
    """A thread's line of ten points is stored as three shifted runs of eight
    for each (dz, dy) it serves; read as the MMA reads it (8-point groups SBO
    apart, taps 16 B apart), element (m, t) is the neighbour of point m at tap t."""
    rng = np.random.default_rng(4)
    field = rng.standard_normal((6, 10, 18))
    w = rng.standard_normal((27, CH))
    smem = np.full(4 * K1_PLANE // 2, np.nan)                          # two-byte elements
    for g in range(4 * 16):                                            # the zero taps
        at = (g * K1_GROUP + 27 * 16) // 2
        smem[at:at + 40] = 0.0
    for line in range(120):
        half, hy, hz = line & 1, (line >> 1) % 10, (line >> 1) // 10
        v = field[hz, hy, 8 * half:8 * half + 10]
        for dz in range(3):
            for dy in range(3):
                oz, oy = hz - dz, hy - dy
                if not (0 <= oz < 4 and 0 <= oy < 8):
                    continue
                for dx in range(3):
                    at = (oz * K1_PLANE + (2 * oy + half) * K1_GROUP + (dz * 9 + dy * 3 + dx) * 16) // 2
                    assert np.isnan(smem[at:at + 8]).all()             # nobody else's
                    smem[at:at + 8] = v[dx:dx + 8]
    for oz in range(4):
        A = np.array([[smem[(oz * K1_PLANE + kh * 256 + (m >> 3) * K1_GROUP + k * 16) // 2 + (m & 7)]
                       for kh in range(2) for k in range(16)] for m in range(128)])
        got = (A[:, :27] @ w).reshape(8, 16, CH)
        want = np.zeros((8, 16, CH))
        for t in range(27):
            dz, dy, dx = t // 9, (t // 3) % 3, t % 3
            want += field[oz + dz, dy:8 + dy, dx:16 + dx][..., None] * w[t]
        assert not A[:, 27:].any()
        assert np.allclose(got, want, rtol=1e-12, atol=1e-12)


# ---- weight gradient (k_conv16_wgrad): plain bricks, a tap is a start address

WX, WLINES, WZ = 16, 3, 8
ROW_A, ROW_B = (WX + 2) * 8, WX * 8                                    # elements of one line of one 8-channel half
PLANE_A, PLANE_B = (WLINES + 2) * 2 * ROW_A, WLINES * 2 * ROW_B
WN = WLINES * CH


def test_weight_gradient_unit_equals_the_direct_sums():
    rng = np.random.default_rng(5)
    x = rng.standard_normal((WZ + 2, WLINES + 2, WX + 2, CH))
    g = rng.standard_normal((WZ, WLINES, WX, CH))
    # [plane][line][half][x][8 channels]; the bytes behind the last plane are read, and ignored
    sa = np.concatenate([x.reshape(WZ + 2, WLINES + 2, WX + 2, 2, 8).transpose(0, 1, 3, 2, 4).ravel(),
                         g.reshape(WZ, WLINES, WX, 2, 8).transpose(0, 1, 3, 2, 4).ravel()])
    off_b = (WZ + 2) * PLANE_A
    k = np.arange(WX)[:, None]
    m = np.arange(128)[None, :]
    D = np.full((128, 9 * WN), np.nan)
    started = set()
    for i in range(WZ + 2):
        q = (i + 2) % (WZ + 2)
        lo, hi = (2 - q if q < 2 else 0), (WZ + 1 - q if q > WZ - 1 else 2)
        n = np.arange((hi - lo + 1) * WN)[None, :]
        for t in range(3):
            a = sa[q * PLANE_A + t * 8 + (m >> 3) * ROW_A + k * 8 + (m & 7)]
            b = sa[off_b + (q - 2 + lo) * PLANE_B + (n >> 3) * ROW_B + k * 8 + (n & 7)]
            cols = slice((3 * t + lo) * WN, (3 * t + hi + 1) * WN)
            if i == 0:
                assert (lo, hi) == (0, 2)
                D[:, cols] = a.T @ b
                started.add(t)
            else:
                D[:, cols] += a.T @ b
    assert started == {0, 1, 2}
    for t in range(27):
        dz, dy, dx = t // 9 - 1, (t // 3) % 3 - 1, t % 3 - 1
        block = 3 * (dx + 1) + 1 - dz
        got = sum(D[(dy + 1 + r) * CH:(dy + 2 + r) * CH, block * WN + r * CH:block * WN + (r + 1) * CH]
                  for r in range(WLINES))
        want = np.einsum("zyxi,zyxo->io", x[1 + dz:1 + dz + WZ, 1 + dy:1 + dy + WLINES, 1 + dx:1 + dx + WX], g)
        assert np.allclose(got, want, rtol=1e-11, atol=1e-11)
