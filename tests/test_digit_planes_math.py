"""Host restatement of the digit products (csrc/oz.cuh): the balanced base-256 digits and the exponent margin they
need, the size of what the 36 kept digit pairs leave out, and the memory order of the planes."""
import math
from fractions import Fraction

import numpy as np
import pytest


def exponent(x: float) -> int:
    x *= 1.005
    return -500 if x == 0.0 else max(-500, math.frexp(x)[1])


def digits(x: float, e: int) -> list:
    """Eight signed digits, most significant first, of round(x 2^(63 - e)) (ties to even in the lower word)."""
    v = Fraction(x) * Fraction(2) ** (63 - e)
    hi = round(Fraction(x) * Fraction(2) ** (31 - e))
    lo = round((v / 2 ** 32 - hi) * 2 ** 32)
    u = (hi * 2 ** 32 + lo + 0x8080808080808080) % 2 ** 64
    return [((u >> (8 * (7 - i))) & 255) - 128 for i in range(8)]


def value(d: list, e: int) -> Fraction:
    return sum(Fraction(di) * 256 ** (7 - i) for i, di in enumerate(d)) * Fraction(2) ** (e - 63)


@pytest.mark.parametrize("x", [1.0, -1.0, 0.0, 0.995, -0.995, 0.9949, 2.0 ** -60, -(2.0 ** -64), 1.0 - 2.0 ** -53,
                               -(1.0 - 2.0 ** -53), 0.5, -0.5, 127.4 / 128, 1e-300, 3.3e100, -7.7e-90])
def test_digits_give_the_number_back(x):
    e = exponent(abs(x))
    d = digits(x, e)
    assert all(-128 <= t <= 127 for t in d)
    assert abs(value(d, e) - Fraction(x)) <= Fraction(2) ** (e - 64)


def test_digits_random_rows_share_an_exponent():
    rng = np.random.default_rng(3)
    row = rng.standard_normal(200) * np.exp(-rng.uniform(0, 40, 200))
    e = exponent(float(np.abs(row).max()))
    for x in row:
        assert abs(value(digits(float(x), e), e) - Fraction(float(x))) <= Fraction(2) ** (e - 64)


def test_kept_pairs_and_the_square_term():
    """sum_k x y from the pairs i + j <= 7; for x == y the pair (4, 4) is the part that does not average out."""
    rng = np.random.default_rng(4)
    K = 400
    x, y = rng.standard_normal(K), rng.standard_normal(K)
    ex, ey = exponent(float(np.abs(x).max())), exponent(float(np.abs(y).max()))
    dx = np.array([digits(float(v), ex) for v in x])
    dy = np.array([digits(float(v), ey) for v in y])

    def product(a, b, ea, eb, square=False):
        s = 0
        for i in range(8):
            for j in range(8 - i):
                s += int((a[:, i] * b[:, j]).sum()) * 256 ** (14 - i - j)
        if square:
            s += int((a[:, 4] ** 2).sum()) * 256 ** 6
        return Fraction(s) * Fraction(2) ** (ea + eb - 126)

    exact = sum(Fraction(float(a)) * Fraction(float(b)) for a, b in zip(x, y))
    # dropped: the 28 pairs beyond i + j = 7, seven of them at weight 256^6 with digits of RMS 74 (six sigma), the
    # rest 256 times smaller, and the rounding of the digits
    bound = 6 * math.sqrt(7 * K) * 74 ** 2 * 2.0 ** (48 + ex + ey - 126) * 1.05 + K * 2.0 ** (ex + ey - 63)
    assert abs(float(product(dx, dy, ex, ey) - exact)) <= bound
    exact = sum(Fraction(float(a)) ** 2 for a in x)
    with_square = abs(float(product(dx, dx, ex, ex, True) - exact))
    # the six pairs besides (4, 4) come twice each: sqrt(2) on their sum
    assert with_square <= math.sqrt(2) * bound
    assert abs(float(product(dx, dx, ex, ex) - exact)) > 3 * with_square


@pytest.mark.parametrize("rows,k,rt", [(1, 1, 128), (130, 33, 128), (300, 64, 128), (80, 47, 64), (64, 32, 64), (48, 31, 64)])
def test_plane_order_is_a_bijection(rows, k, rt):
    kb = -(-k // 32)
    tile = kb * 8 * rt * 32

    def tile_rows(r):
        left = -(-rows // 16) * 16 - r // rt * rt
        return rt if rt == 128 or left >= rt else left

    def at(r, kk, d):
        i, j = r % rt, kk % 32
        return (r // rt * tile + kk // 32 * (8 * tile_rows(r) * 32) + i // 8 * 256 + j // 16 * 128 + i % 8 * 16 + j % 16 +
                d * tile_rows(r) * 32)

    seen = {at(r, kk, d) for r in range(rows) for kk in range(kb * 32) for d in range(8)}
    assert len(seen) == rows * kb * 32 * 8
    assert max(seen) < -(-rows // rt) * tile
    # a K block of a tile is one run over all planes, and every group of eight K bytes one aligned run
    for r in range(0, rows, 7):
        assert at(r, 0, 0) % 8 == 0 and all(at(r, q, 3) == at(r, 0, 3) + q for q in range(8))
