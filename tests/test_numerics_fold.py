"""Host models of the arithmetic of the grouped scan's FP64 sums as it runs (rf_device.cuh), checked
against exact rational arithmetic, with numpy's float32 for the device's round-to-nearest operations:

* rf_df_split_in: a double of the range -> two floats, the low one rounded: |v - (hi + lo)| <= 2^-47 v.
* rf_tf_add2 / rf_tf2_to_f64: double-floats summed as three floats within 2^-58, and the double nearest
  the sum, the low part's sign and the carry into the next power of two included.
"""
import struct
from fractions import Fraction

import numpy as np
import pytest

from test_numerics_model import F32, _f32, _words, df_add


def bits32(x):
    return struct.unpack("<I", struct.pack("<f", x))[0]


def df_in(v):
    return ((_words(v)[0] - (920 << 20)) & 0xFFFFFFFF) < (194 << 20)


def split_in(v):
    """rf_df_split_in<Z = true>."""
    h, l = _words(v)
    hb = ((((h - (896 << 20)) & 0xFFFFFFFF) << 3) | (l >> 29)) & 0xFFFFFFFF
    c = ((hb & 0x7F800000) - (23 << 23)) & 0xFFFFFFFF
    lo = F32(_f32(c + (((l & 0x1FFFFFFF) + 32) >> 6)) - _f32(c))
    return _f32(0 if h == 0 else hb), lo


def two_sum(a, b):
    s = F32(a + b)
    bb = F32(s - a)
    return s, F32(F32(a - F32(s - bb)) + F32(b - bb))


def tf_add(a, b):
    """rf_tf_add2, one of its two sums."""
    h, e1 = two_sum(a[0], b[0])
    m, e2 = two_sum(a[1], b[1])
    m, e3 = two_sum(m, e1)
    return h, m, F32(F32(a[2] + b[2]) + F32(e2 + e3))


def rint32(x):
    """__float2int_rn."""
    return int(np.rint(F32(x)))


def to_f64(hi, mid, lo=F32(0)):
    """rf_tf_to_f64."""
    hb = bits32(hi)
    eh, half = hb >> 23, 1 if (hb & 0x7FFFFF) == 0 and mid < 0 else 0
    small = eh < 64
    s1 = F32(2.0 ** 60) if small else F32(1)
    s2 = _f32((306 + half - eh - (60 if small else 0)) << 23)
    with np.errstate(under="ignore"):
        x, y = F32(F32(mid * s1) * s2), F32(F32(lo * s1) * s2)
    i = rint32(x)
    k = rint32(F32(F32(x - F32(i)) + y))
    m = (((hb & 0x7FFFFF) | 0x800000) << (29 + half)) + i + k
    if hb == 0:
        return 0.0
    assert 2 ** 52 <= m <= 2 ** 53, (hi, mid, lo)
    return struct.unpack("<d", struct.pack("<Q", ((eh + 896 - half) << 52) + (m - (1 << 52))))[0]


def tf_to_f64(a):
    """rf_tf2_to_f64, one of its two sums."""
    h, m = two_sum(a[0], a[1])
    m, l = two_sum(m, a[2])
    h, m = two_sum(h, m)
    return to_f64(h, m, l)


def exact(parts):
    return sum(Fraction(float(p)) for p in parts)


def doubles(n, seed):
    rng = np.random.default_rng(seed)
    v = list(rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-103, 91, n))
    for e in (-103, -64, -63, -62, -1, 0, 1, 52, 90):
        p = 2.0 ** e
        v += [p, np.nextafter(p, np.inf), p * (1 + 2.0 ** -23), p * (2 - 2.0 ** -23), p * (1 + 2.0 ** -24), np.nextafter(2 * p, 0)]
        v += [p * (1 + 2.0 ** -23 - 2.0 ** -k) for k in range(24, 53)]  # low parts up to the next unit of hi
    return [float(x) for x in v if df_in(float(x))]


def test_rounding_split():
    for v in doubles(4000, 1):
        hi, lo = split_in(v)
        assert abs(Fraction(v) - exact((hi, lo))) <= Fraction(v) / 2 ** 47, v
        assert 0 <= lo and Fraction(float(lo)) <= Fraction(float(hi)) / 2 ** 23
    assert split_in(0.0) == (0, 0)
    for v in [-1.0, -0.0, 0.0, 5e-324, np.nextafter(2.0 ** -103, 0), 2.0 ** 91, float("inf"), float("nan"), -2.0 ** -103]:
        assert not df_in(v), v
    assert df_in(2.0 ** -103) and df_in(np.nextafter(2.0 ** 91, 0))


def test_a_pair_becomes_the_nearest_double():
    rng = np.random.default_rng(2)
    checked = 0
    for v in doubles(4000, 2) + [2.0 ** e for e in range(-103, 120)]:
        hi, lo = split_in(v) if v < 2.0 ** 91 else (F32(v), F32(0))
        unit = float(hi) * 2.0 ** -24  # about half a unit of hi's last place
        lows = [lo, F32(0)] + [F32(s * unit * x) for s in (1, -1) for x in (0.49, 2.0 ** -4, 2.0 ** -22, 2.0 ** -28, 2.0 ** -29, 2.0 ** -30)]
        lows += [F32(x) for x in rng.uniform(-0.5, 0.5, 4) * unit]
        for x in lows:
            h, l = two_sum(hi, x)
            if not 2.0 ** -103 <= h < 2.0 ** 127:
                continue
            got, want = Fraction(to_f64(h, l)), exact((h, l))
            assert got == Fraction(float(want)) or abs(got - want) == abs(Fraction(float(want)) - want), (v, x)
            checked += 1
    assert checked > 40_000
    assert to_f64(F32(0), F32(0)) == 0.0


@pytest.mark.parametrize("rows", [1, 2, 8, 32])
@pytest.mark.parametrize("kind", ["whole", "uniform", "spread", "zeros", "tiny"])
def test_sums_over_the_threads_of_a_block(kind, rows):
    # 512 threads of `rows` rows each: 16 warps' slots to a lane in four chains, the chains two by two, the
    # lanes by halves, as the kernel adds them
    rng = np.random.default_rng(rows)
    n = 512 * rows
    v = {"whole": lambda: rng.integers(1, 2 ** 44 // rows, n).astype(np.float64), "uniform": lambda: rng.uniform(900.0, 105000.0, n),
         "spread": lambda: rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-100, 80, n),
         "zeros": lambda: np.where(rng.random(n) < 0.9, 0.0, rng.uniform(0.0, 0.1, n)),
         "tiny": lambda: rng.uniform(1.0, 2.0, n) * 2.0 ** -103}[kind]().reshape(512, rows)
    slots = []
    for t in v:
        a = (F32(0), F32(0))
        for x in t:
            a = df_add(*a, *split_in(float(x)))
        slots.append(a)
    want = sum(exact(s) for s in slots)  # the slots' own exact sum
    lanes = []
    for lane in range(32):
        a = [(*slots[lane + 32 * k], F32(0)) for k in range(4)]
        for k in range(4, 16):
            a[k % 4] = tf_add(a[k % 4], (*slots[lane + 32 * k], F32(0)))
        a = [tf_add(a[0], a[2]), tf_add(a[1], a[3])]
        lanes.append(tf_add(a[0], a[1]))
    for off in (16, 8, 4, 2, 1):
        lanes = [tf_add(lanes[i], lanes[i + off]) for i in range(off)]
    assert abs(exact(lanes[0]) - want) <= want / 2 ** 58
    got = Fraction(tf_to_f64(lanes[0]))
    assert abs(got - want) <= want / 2 ** 53 + want / 2 ** 58  # one rounding to a double
    if kind == "whole":
        assert want == int(v.sum()) and got == want
