"""CPU restatement of the FP64 digit products' integers (eight 8-bit digits of
62 bits, exact levels of 128 rows, sums hi 2^20 + lo): the digits give the
value back, the level sums stay exact in FP32, the 64-bit sums cannot
overflow, and the leading bits round as the whole sum does."""
import numpy as np

BITS, BASE, DIG, ROWS, FOLDS = 62, 8, 8, 128, 64


def _int32(x):
    return ((x + (1 << 31)) & 0xFFFFFFFF) - (1 << 31)


def _digits(w):
    hh = (w + (1 << 31)) >> 32
    h, l = _int32(hh), _int32(w - (hh << 32))
    d = [0] * DIG
    for t in range(3):
        sh = BASE * (3 - t)
        d[t] = ((h >> (sh - 1)) + 1) >> 1
        h = _int32(h - (d[t] << sh))
        d[4 + t] = ((l >> (sh - 1)) + 1) >> 1
        l = _int32(l - (d[4 + t] << sh))
    d[3], d[7] = h, l
    return d


def _samples():
    rng = np.random.default_rng(1)
    edge = [0, 1, 127, 128, 129, 2 ** 31 - 1, 2 ** 31, 2 ** 31 + 1,
            2 ** 32 - 1, 2 ** 62 - 2 ** 9, 2 ** 62 - 1, 2 ** 62]
    rand = [int(v) >> int(s) for v, s in
            zip(rng.integers(0, 2 ** 62, 4000), rng.integers(0, 60, 4000))]
    return [s * v for v in edge + rand for s in (1, -1)]


def test_digits_give_the_value_back():
    for w in _samples():
        d = _digits(w)
        assert sum(a << (BASE * (DIG - 1 - t)) for t, a in enumerate(d)) == w
        assert abs(d[0]) <= 64 and max(map(abs, d)) <= 128


def test_levels_are_exact_and_sums_fit():
    top = [64] + [128] * (DIG - 1)
    level = [ROWS * sum(top[t] * top[l - t] for t in range(l + 1))
             for l in range(DIG)]
    assert max(level) <= 2 ** 24  # integers that FP32 holds
    for a, b in ((0, 1), (2, 3)):  # combined in 32 bits
        assert level[a] * 256 + level[b] < 2 ** 31
    low = ((level[4] * 256 + level[5]) << 16) + level[6] * 256 + level[7]
    assert low + 2 ** 20 < 2 ** 63
    hi = ((level[0] * 256 + level[1]) << 28) + (
        (level[2] * 256 + level[3]) << 12) + (low >> 20) + 1
    assert FOLDS * hi < 2 ** 63


def test_leading_bits_round_as_the_sum():
    rng = np.random.default_rng(2)
    for _ in range(4000):
        hi = int(rng.integers(-2 ** 62, 2 ** 62)) >> int(rng.integers(0, 62))
        lo = int(rng.integers(-2 ** 19, 2 ** 19))
        m = hi ^ (hi >> 63)
        sh = min(max(64 - m.bit_length() - 2, 0), 20)
        lead = (hi << sh) + (lo >> (20 - sh))
        assert abs(lead) < 2 ** 63
        whole = (hi << 20) + lo
        err = abs(int(float(lead)) * 2 ** (20 - sh) - whole)
        # half a unit in the last place, and what the shift cut off
        assert err <= 2 ** max(whole.bit_length() - 54, 0) * 1.01
