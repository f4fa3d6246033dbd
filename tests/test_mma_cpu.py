"""numpy model of the tensor-core decode matvec (xalm_b200/csrc/matvec_mma.cuh) and of its weight layout
(xalm_b200/csrc/frag_layout.cuh), run on the CPU.

The kernel feeds mma.sync.m16n8k32.s8.u8.s32 (u8.u8 for the formats with a minimum) with quants times MUL as A and, as B, the three unsigned limbs of the
OFFSET activations X' = X + 2^23 plus a column of ones; the accumulators start at zero.  This file restates that arithmetic and checks the claims of the kernel's header:
  * the bytes that a record's stored quant becomes are MUL * quant, signed, for every code;
  * 65536 * v(l0', ones) + v(l1', l2') == MUL * sum_k q_k * X_k exactly;
  * every intermediate fits int32;
  * a one-hot x gives back d * q (+ m) bit for bit, with the factors 65536 and 1 / MUL applied at a tile's end;
and for the layout: the (row, element) -> byte map of a record is a bijection that puts the mma's A fragment of lane t at
bytes [16 t, 16 t + 16) (8-bit) / [8 t, 8 t + 8) (4-bit), with the two rows of a GLU pair in the same lane.
The GPU side of the same checks is tests/test_gpu_formats.py (one-hot bit exactness, random x against the oracle).
"""
import numpy as np
import pytest

F32 = np.float32


# format -> (MUL, has a minimum, what the kernel makes of a stored code as the byte fed to the mma, the code's quant)
def nibble_up(u):
    return ((u << 4) & 0xF0) ^ 0x80           # Q4_0: a nibble in the byte's upper half, its top bit turned


FORMATS = {
    "q8_0": (1, False, lambda u: u ^ 0x80, lambda u: u - 128, 256),
    "q4_0": (16, False, nibble_up, lambda u: u - 8, 16),
    "q5_0": (8, False, lambda u: ((u << 3) & 0xFF) ^ 0x80, lambda u: u - 16, 32),
    "q4_1": (1, True, lambda u: u, lambda u: u, 16),
    "q5_1": (1, True, lambda u: u, lambda u: u, 32),
}


def operand(fmt, u):
    """The bytes that codes u become, as the mma reads them: signed, or unsigned where there is a minimum."""
    b = FORMATS[fmt][2](np.asarray(u, dtype=np.int64)) & 0xFF
    return b if FORMATS[fmt][1] else np.where(b >= 128, b - 256, b)


@pytest.mark.parametrize("fmt", FORMATS)
def test_the_byte_of_every_code_is_its_quant_times_mul(fmt):
    mul, _, _, quant, n = FORMATS[fmt]
    u = np.arange(n)
    assert np.array_equal(operand(fmt, u), mul * quant(u))


def stage_block(x):
    """xm_store_group8 over one 32-element block: X, the offset limbs l0' l1' l2' (each 0..255), dx."""
    x = np.asarray(x, dtype=F32)
    mb = int(np.max(x.view(np.uint32) & 0x7FFFFFFF))
    eb = mb >> 23
    live = 40 <= eb < 255
    sc = np.array([(276 - eb) << 23], np.uint32).view(F32)[0] if live else F32(0)
    dx = np.array([(eb - 22) << 23], np.uint32).view(F32)[0] if live else F32(0)
    with np.errstate(invalid="ignore"):
        prod = np.nan_to_num((x * sc).astype(F32), nan=0.0)            # __float2int_rn(NaN) = 0 (inf * 0 in a dropped block)
    X = np.minimum(np.rint(prod).astype(np.int64), 8388607)
    Xo = X + 8388608
    assert Xo.min() >= 0 and Xo.max() < 1 << 24
    return X, np.stack([(Xo >> 16) & 255, (Xo >> 8) & 255, Xo & 255]), dx


def mma_block(a, limbs):
    """One record column of the mma for one row: the accumulators of the four used B columns, from zero -> (v01, v23)."""
    c_l2, c_l1, c_l0, c_one = (int(np.dot(a, limbs[2])), int(np.dot(a, limbs[1])), int(np.dot(a, limbs[0])), int(a.sum()))
    for c in (c_l2, c_l1, c_l0, c_one):
        assert abs(c) < 2 ** 31
    v01 = 256 * c_l1 + c_l2          # lane position 0: columns (l2', l1')
    v23 = c_l0 - 128 * c_one         # lane position 1: columns (l0', ones); 128 * 65536 = 2^23 removes the offset
    assert abs(256 * c_l1) < 2 ** 31 and abs(128 * c_one) < 2 ** 31 and abs(v01) < 2 ** 31 and abs(v23) < 2 ** 31
    return v01, v23


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("scale", [1e-12, 1.0, 250.0])
def test_offset_limb_mma_is_the_exact_integer_dot_product(fmt, scale):
    mul, _, _, quant, n = FORMATS[fmt]
    rng = np.random.default_rng(n * 7 + mul)
    for trial in range(40):
        x = (rng.standard_normal(32) * scale).astype(F32)
        u = rng.integers(0, n, 32)
        if trial < 4:                                   # the largest sums: every element at the block's maximum, the quants at either end
            x[:] = (1 if trial & 1 else -1) * np.abs(x).max()
            u[:] = n - 1 if trial & 2 else 0
        X, limbs, dx = stage_block(x)
        v01, v23 = mma_block(operand(fmt, u), limbs)
        assert 65536 * v23 + v01 == mul * int(np.dot(quant(u), X))


def test_dead_and_nonfinite_blocks_contribute_nothing():
    for x in (np.zeros(32, F32), np.full(32, 1e-30, F32), np.array([np.inf] + [1.0] * 31, F32)):
        X, limbs, dx = stage_block(x)
        assert dx == 0 and np.all(X == 0)
        v01, v23 = mma_block(operand("q8_0", np.full(32, 200)), limbs)
        assert 65536 * v23 + v01 == 0                   # and dx = 0 multiplies either lane's part


@pytest.mark.parametrize("fmt", FORMATS)
def test_one_hot_returns_the_dequantised_weight_bit_for_bit(fmt):
    mul, has_min, _, quant, n = FORMATS[fmt]
    rng = np.random.default_rng(3)
    for _ in range(200):
        j = int(rng.integers(0, 32))
        x = np.zeros(32, F32)
        x[j] = 1.0
        X, limbs, dx = stage_block(x)
        u = rng.integers(0, n, 32)
        d = F32(np.float16(rng.standard_normal() * 0.1))
        m = F32(np.float16(rng.standard_normal())) if has_min else None
        v01, v23 = mma_block(operand(fmt, u), limbs)
        # either lane adds float(v) * (d * dx); at the tile's end lane position 0 is multiplied by 1 / MUL, 1 by 65536 / MUL, and the two are added
        y0 = F32(F32(v01) * F32(d * dx))
        y1 = F32(F32(v23) * F32(d * dx))
        if has_min:
            sx = F32(F32(int(X.sum())) * dx)
            assert sx == 1.0
            y0 = F32(np.float64(m) * np.float64(sx) + np.float64(y0))
        y = F32(F32(y0 * F32(1.0 / mul)) + F32(y1 * F32(65536.0 / mul)))
        want = F32(F32(d * F32(int(quant(u[j])))) + (m if has_min else F32(0)))   # quants.py: d * q (+ m), one rounding
        assert y.view(np.uint32) == want.view(np.uint32) or (y == 0 and want == 0)


# ---- layout (frag_layout.cuh) -------------------------------------------------------------------------------------------
def rec_offset_8bit(row, kk):
    g, hi = row % 8, row // 8
    tig, e, j = (kk % 16) // 4, kk % 4, (kk // 16) * 2 + hi
    return (g * 4 + tig) * 16 + j * 4 + e


def rec_offset_4bit(row, kk):
    g, hi = row % 8, row // 8
    tig, e, half = (kk % 16) // 4, kk % 4, kk // 16
    return (g * 4 + tig) * 8 + half * 4 + e, hi     # (byte, nibble)


def test_record_layout_is_the_mma_a_fragment():
    seen8, seen4 = set(), set()
    for row in range(16):
        for kk in range(32):
            o = rec_offset_8bit(row, kk)
            assert 0 <= o < 512 and o not in seen8
            seen8.add(o)
            b, nib = rec_offset_4bit(row, kk)
            assert 0 <= b < 256 and (b, nib) not in seen4
            seen4.add((b, nib))
            # PTX m16n8k32 A fragment: byte i of lane t = 4 * groupID + threadID_in_group holds
            #   row = groupID (+ 8 for i in 4..7, 12..15), col = 4 * threadID_in_group + (i & 3) (+ 16 for i >= 8)
            t, i = o // 16, o % 16
            assert row == t // 4 + (8 if (i // 4) % 2 else 0) and kk == 4 * (t % 4) + (i & 3) + (16 if i >= 8 else 0)
            t4, i4 = b // 8, b % 8
            assert row % 8 == t4 // 4 and row // 8 == nib and kk == 4 * (t4 % 4) + (i4 & 3) + (16 if i4 >= 4 else 0)
    assert len(seen8) == 512 and len(seen4) == 512


def frag_virtual_row(glu_half, r):
    if not glu_half:
        return r
    o = r if r < glu_half else r - glu_half
    return (o // 8) * 16 + (0 if r < glu_half else 8) + o % 8


def test_glu_pairs_share_a_lane():
    H = 64
    vr = [frag_virtual_row(H, r) for r in range(2 * H)]
    assert sorted(vr) == list(range(2 * H))                       # a permutation of the stacked gate|up rows
    for o in range(H):
        a, b = vr[o], vr[H + o]
        assert a // 16 == b // 16 and b - a == 8                  # same tile, rows g and g + 8: registers (c0,c1) and (c2,c3) of one lane
        assert a // 16 * 8 + a % 8 == o                           # the epilogue's output index row0 / 2 + lane
