"""The quotients of the register-blocked Horn-Schunck sweep (hr_div and hr_div_wide in csrc/hsweep.cuh),
restated with exactly rounded float32 operations: the correctly rounded num / den (numpy's float32
division) over the ranges their comments state, with operands next to rounding midpoints and quotients
on the midpoints of the subnormal numbers."""
import numpy as np

F = np.float32


def fma(a, b, c):
    """float32 fma: the product is exact in float64, the sum is rounded to odd there and then to float32
    (53 bits against 24: the second rounding is the only one)."""
    p = a.astype(np.float64) * b.astype(np.float64)
    c = c.astype(np.float64)
    s = p + c
    t = s - p
    e = (p - (s - t)) + (c - t)  # s + e is the sum
    bits = s.view(np.int64)
    odd = (e != 0) & (bits & 1 == 0)
    toward = np.where((e > 0) == (s > 0), bits + 1, bits - 1)
    return np.where(odd, toward, bits).view(np.float64).astype(F)


def hr_div(num, den, y):
    q = num * y
    q = fma(fma(-q, den, num), y, q)
    return fma(fma(-q, den, num), y, q)


def hr_div_wide(num, den, y):
    tiny = np.abs(num) < F(2.0 ** -60)
    up = np.where(tiny, F(2.0 ** 64), F(1))
    n = num * up
    q = hr_div(n, den, y)
    der = q * np.where(tiny, F(2.0 ** -64), F(1))
    e, r = fma(der, up, -q), fma(-q, den, n)
    down, more = (e == F(2.0 ** -86)) & (r < 0), (e == -F(2.0 ** -86)) & (r > 0)
    return np.where(down, der - F(2.0 ** -149), np.where(more, der + F(2.0 ** -149), der)).astype(F)


def check(f, num, den):
    with np.errstate(all="ignore"):
        want = num / den
        got = f(num, den, F(1) / den)
    bad = want.view(np.uint32) != got.view(np.uint32)
    assert not bad.any(), (num[bad][:4], den[bad][:4], want[bad][:4], got[bad][:4])


def mantissas(rng, n, e0, e1):
    """Full-precision numbers of either sign with exponents e0 .. e1 - 1."""
    m = np.ldexp(1.0 + rng.integers(0, 1 << 23, n) / 2.0 ** 23, rng.integers(e0, e1, n))
    return m * rng.choice([-1.0, 1.0], n)


def near_midpoints(rng, den, e0, e1):
    """Numerators whose quotient by den lies next to the middle of two float32 numbers."""
    q = mantissas(rng, den.size, e0, e1).astype(F)
    mid = (q.astype(np.float64) + np.nextafter(q, F(np.inf)).astype(np.float64)) / 2
    base = (den.astype(np.float64) * mid).astype(F)
    return [(base.view(np.int32) + np.int32(k)).view(F) for k in range(-2, 3)]


def test_refined_quotient():
    rng = np.random.default_rng(1)
    n = 1 << 19
    den = np.abs(mantissas(rng, n, -40, 40)).astype(F)
    check(hr_div, mantissas(rng, n, -80, 60).astype(F), den)
    check(hr_div, np.zeros(n, F), den)
    lo, hi = F(2.0 ** -80), F(2.0 ** 60)
    for d in (den, np.full(n, np.nextafter(F(2), F(0))), (441 + rng.integers(0, 1 << 16, n) / 16).astype(F)):
        for num in near_midpoints(rng, d, -30, 20):
            ok = (np.abs(num) >= lo) & (np.abs(num) <= hi)
            check(hr_div, num[ok], d[ok])


def test_wide_quotient():
    rng = np.random.default_rng(2)
    n = 1 << 19
    den = np.abs(mantissas(rng, n, -40, 40)).astype(F)
    for num in (mantissas(rng, n, -149, 60), mantissas(rng, n, -149, -100), np.ldexp(rng.integers(-4096, 4097, n), -149)):
        num = num.astype(F)
        num[num == 0] = 0  # +0; -0 is left to the divide
        check(hr_div_wide, num, den)
    for num in near_midpoints(rng, den, -90, -20):
        ok = num != 0
        check(hr_div_wide, num[ok], den[ok])


def test_wide_quotient_on_subnormal_midpoints():
    """num = den * M * 2^-150 with M odd is exact for short den: ties, and their neighbours by one unit."""
    rng = np.random.default_rng(3)
    n = 1 << 19
    den = (2.0 * rng.integers(1, 1 << 10, n)).astype(F)
    m = 2 * rng.integers(0, 1 << 12, n) + 1
    tie = np.ldexp(den.astype(np.float64) * m, -150)
    for k in (-1, 0, 1):
        num = ((tie + np.ldexp(float(k), -149)) * rng.choice([-1.0, 1.0], n)).astype(F)
        ok = num != 0
        check(hr_div_wide, num[ok], den[ok])


def hq_div(num, den):
    """hq_div: the product with the float64 reciprocal, rounded to a multiple of 2^-177 where it is subnormal."""
    q = num.astype(np.float64) * (1.0 / den.astype(np.float64))
    c = 1.5 * 2.0 ** -125
    s = (q + c) - c
    return np.where((np.abs(q) >= 2.0 ** -151) & (np.abs(q) < 2.0 ** -126), s, q).astype(F)


def test_float64_quotient_of_subnormal_results():
    """Quotients on and next to the midpoints of the subnormal numbers, random ones, and all the short
    numerators a diffusing flow ends in."""
    rng = np.random.default_rng(4)
    n = 1 << 19
    f = lambda num, den, y: hq_div(num, den)  # noqa: E731
    for den in ((2.0 * rng.integers(1, 1 << 10, n)).astype(F), (441 + rng.integers(0, 1 << 16, n) / 16).astype(F),
                np.abs(mantissas(rng, n, -30, 60)).astype(F)):
        m = 2 * rng.integers(0, 1 << 12, n) + 1
        tie = np.ldexp(den.astype(np.float64) * m, -150)
        for k in (-1, 0, 1):
            check(f, ((tie + np.ldexp(float(k), -149)) * rng.choice([-1.0, 1.0], n)).astype(F), den)
        check(f, np.ldexp(rng.integers(-4096, 4097, n).astype(float), -149).astype(F), den)
        check(f, mantissas(rng, n, -149, -90).astype(F), den)
        check(f, mantissas(rng, n, -60, 60).astype(F), den)
