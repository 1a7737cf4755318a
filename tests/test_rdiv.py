"""The shared-reciprocal root and divisions of the FP64 walk (csrc/nb_rdiv.cuh), no GPU.

The header uses only fma, * and integer operations after the reciprocal estimate, so a host
build of it computes what the device computes from an estimate of the same quality (the host's
keeps 20 bits of 1/sqrt(s), as the device's instruction does).  Every result must equal the IEEE
operator's, bit for bit: on random operands over the exponent ranges the walk admits, and on
roots and quotients constructed to lie next to a rounding boundary.
"""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "milkywayathome_client_b200", "csrc")
SRC = r'''
#include "nb_rdiv.cuh"
extern "C" void radial(const double* s, const double* m, const double* a, int n, double* out)
{
    for (int i = 0; i < n; ++i) {
        double y;
        const double r = nb_sqrt_recip(s[i], nb_rsqrt_estimate(s[i]), y);
        const double z = nb_recip_step(s[i], y * y);
        const double t = (s[i] * s[i]) * r;
        out[5 * i] = r;
        out[5 * i + 1] = nb_quot(m[i], r, y);
        out[5 * i + 2] = nb_quot(nb_quot(m[i], r, y), s[i], z);
        out[5 * i + 3] = nb_recip_step(t, nb_recip_step(t, (z * z) * y));
        out[5 * i + 4] = nb_quot(a[i], s[i], z);
    }
}
extern "C" void reciprocals(const double* s, int n, double* out)
{
    for (int i = 0; i < n; ++i) {
        double y;
        const double r = nb_sqrt_recip(s[i], nb_rsqrt_estimate(s[i]), y);
        out[4 * i] = r;
        out[4 * i + 1] = y;                                 // nearly rounded 1 / r
        out[4 * i + 2] = nb_recip_step(s[i], y * y);        // nearly rounded 1 / s
        out[4 * i + 3] = nb_recip_step(s[i], out[4 * i + 2]);
    }
}
extern "C" void quotients(const double* a, const double* b, const double* y, int n, double* out)
{
    for (int i = 0; i < n; ++i) out[i] = nb_quot(a[i], b[i], y[i]);
}
extern "C" void plummer(const double* s, const double* m, const double* x, const double* a, int n,
                        double* out)
{
    for (int i = 0; i < n; ++i) {
        double y;
        const double r = nb_sqrt_recip(s[i], nb_rsqrt_estimate(s[i]), y);
        out[3 * i] = nb_quot(m[i], r, y);                   // m / sqrt(s)
        out[3 * i + 1] = nb_recip_step(r, y);               // 1 / sqrt(s)
        out[3 * i + 2] = nb_quot(x[i], a[i], 1.0 / a[i]);   // x / a
    }
}
extern "C" void ranges(const double* x, int n, int* out)
{
    for (int i = 0; i < n; ++i)
        out[i] = nb_exp_in<-700, 700>(x[i]) | nb_pos_exp_in<-100, 100>(x[i]) << 1 |
                 nb_near_ones(x[i]) << 2 | nb_is_zero(x[i]) << 3;
}
'''


# operands whose 1 / s, or whose root's reciprocal, one step from a few ulps does not round
HARD_RECIPROCALS = [4663060627120798 * 2.0 ** -53, 8042426583074580 * 2.0 ** -53,
                    float.fromhex("0x1.30a0dd90e13a2p+0"), float.fromhex("0x1.63baaac17d1e2p+1"),
                    float.fromhex("0x1.0499b629293abp+0"), float.fromhex("0x1.0d5f392d40883p+0")]


def hard_roots():
    """Every s in [1, 4) whose root lies within 40 units of 2^-106 / (2 sqrt(s)) of a midpoint m of
    two doubles: with M = 2^53 m odd, s = (M^2 - c) 2^-106 for |c| < 40 (c = 1 mod 8, for M^2 is and s
    is a multiple of 2^-52).  The four roots of M^2 = c mod 2^k follow from those mod 2^(k - 1)."""
    found = []
    for c in range(-39, 40, 8):
        for k, top in ((54, 2.0), (55, 4.0)):       # s below 2: multiples of 2^-52; below 4: of 2^-51
            roots = {1, 3, 5, 7}
            for j in range(4, k + 1):
                roots = {r + h for r in roots for h in (0, 1 << (j - 1))
                         if ((r + h) ** 2 - c) % (1 << j) == 0}
            for M in roots:
                if (1 << 53) < M < (1 << 54):
                    s = (M * M - c) / 2.0 ** 106    # an integer of 53 bits times a power of two
                    assert Fraction(s) == Fraction(M * M - c, 1 << 106) or not top / 2 <= s < top
                    if top / 2 <= s < top:
                        found.append(s)
    return found


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rdiv")
    src = d / "rdiv.cpp"
    src.write_text(SRC)
    so = d / "librdiv.so"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-mfma", "-fPIC", "-shared", "-I", CSRC,
                    str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def _near_ones(x):
    return (x.view(np.uint64) >> np.uint64(32)) & np.uint64(0xfffff) == 0xfffff


def _check(lib, s, m, a):
    s, m, a = (np.ascontiguousarray(x, dtype=np.float64) for x in (s, m, a))
    out = np.empty((len(s), 5))
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (s, m, a)]
    lib.radial(*p, ctypes.c_int(len(s)), out.ctypes.data_as(ctypes.c_void_p))
    r = np.sqrt(s)
    want = np.stack([r, m / r, (m / r) / s, 1.0 / ((s * s) * r), a / s], 1)
    # the walk leaves divisors next to an all-ones significand to the operators (nb_near_ones)
    ones = np.zeros(want.shape, bool)
    ones[:] = _near_ones(s)[:, None]
    ones[:, 3] |= _near_ones((s * s) * r)
    bad = np.nonzero((out.view(np.uint64) != want.view(np.uint64)) & ~ones)
    assert len(bad[0]) == 0, (bad[0][:5], bad[1][:5], out[bad][:5], want[bad][:5])


def _random(rng, n, lo, hi):
    x = np.ldexp(1.0 + rng.integers(0, 1 << 52, n) * 2.0 ** -52, rng.integers(lo, hi, n))
    return x


@pytest.mark.parametrize("seed", range(4))
def test_random_operands(lib, seed):
    rng = np.random.default_rng(seed)
    n = 500_000
    sign = rng.choice([-1.0, 1.0], n)
    _check(lib, _random(rng, n, -100, 100), sign * _random(rng, n, -700, 700),
           -sign * _random(rng, n, -700, 700))
    _check(lib, _random(rng, n, -8, 12), _random(rng, n, -20, 4), sign * _random(rng, n, -40, 20))


def test_operands_next_to_rounding_boundaries(lib):
    """Roots whose square lies next to that of a midpoint of two doubles, and quotients a / s with
    a = round(s q) for a midpoint q, a few ulps around each."""
    rng = np.random.default_rng(9)
    n = 200_000
    k = rng.integers(1 << 52, 1 << 53, n, dtype=np.int64)
    mid = [2 * int(v) + 1 for v in k[:20000]]
    s = []
    for v in mid:
        sq = v * v                                  # (midpoint)^2, 107 or 108 bits
        sh = sq.bit_length() - 53
        for d in (-1, 0, 1, 2):
            s.append(float((sq >> sh) + d) * 2.0 ** (sh - 107 + (sh & 1)))
    s = np.array(s)
    _check(lib, s, np.ones_like(s), np.ones_like(s))
    s = _random(rng, n, -3, 3)
    si = np.ldexp(s, 52 - np.frexp(s)[1] + 1).astype(np.int64)
    a = np.array([float((int(x) * (2 * int(q) + 1) >> 53) + d)
                  for x, q, d in zip(si, k, rng.integers(-1, 3, n))])
    _check(lib, s, a, a)
    # significands of all ones and of zeros, powers of two, neighbours of one
    edge = np.array([1.0, 2.0, 4.0, 2.0 - 2.0 ** -52, 4.0 - 2.0 ** -51, 1.0 + 2.0 ** -52, 3.0,
                     np.nextafter(0.25, 0), np.nextafter(0.5, 1)])
    g = np.array(np.meshgrid(edge, edge, edge)).reshape(3, -1)
    _check(lib, *g)


def test_hard_roots(lib):
    """The only operands the bound on the root leaves open, in several binades."""
    hard = hard_roots()
    assert len(hard) >= 10 and 1.0 + 2.0 ** -52 in hard
    s = np.array([h * 4.0 ** k for h in hard for k in (-50, -26, -3, 0, 1, 17, 49)])
    _check(lib, s, np.ones_like(s), np.full_like(s, 3.0))


def _off(y, b):
    """|y - 1/b| in ulps of 1/b, exactly."""
    inv = 1 / Fraction(b)
    ulp = Fraction(2.0 ** np.floor(np.log2(float(inv)))) / 2 ** 52
    while ulp * 2 ** 52 > inv:
        ulp /= 2
    while ulp * 2 ** 53 <= inv:
        ulp *= 2
    return abs(Fraction(y) - inv) / ulp


def test_reciprocals_are_nearly_rounded(lib):
    """What nb_quot and the second step are given: |y - 1/b| <= (1/2 + 2^-40) ulp, b the root and s;
    a second step then rounds 1 / s.  On random operands and on those where one step does not."""
    rng = np.random.default_rng(3)
    s = np.concatenate([HARD_RECIPROCALS, hard_roots(), _random(rng, 4000, -100, 100)])
    s = s[~_near_ones(s)]
    out = np.empty((len(s), 4))
    lib.reciprocals(s.ctypes.data_as(ctypes.c_void_p), ctypes.c_int(len(s)),
                    out.ctypes.data_as(ctypes.c_void_p))
    assert np.array_equal(out[:, 0], np.sqrt(s)) and np.array_equal(out[:, 3], 1.0 / s)
    bound = Fraction(1, 2) + Fraction(1, 1 << 40)
    for x, (r, y, z, _) in zip(s, out):
        assert _off(y, r) <= bound and _off(z, x) <= bound
    first = out[:len(HARD_RECIPROCALS)]
    assert ((first[:, 2] != 1.0 / s[:len(first)]) | (first[:, 1] != 1.0 / first[:, 0])).any()


def test_quotients_from_either_neighbour(lib):
    """Quotients next to midpoints, divided with the worst nearly rounded reciprocals there are: of
    divisors whose reciprocal lies next to a midpoint, both neighbours of it."""
    rng = np.random.default_rng(4)
    b = np.array(HARD_RECIPROCALS[:4])
    out = np.empty((4, 4))
    lib.reciprocals(b.ctypes.data_as(ctypes.c_void_p), ctypes.c_int(4),
                    out.ctypes.data_as(ctypes.c_void_p))
    bound = Fraction(1, 2) + Fraction(1, 1 << 40)
    tried = 0
    for x in b:
        ys = [y for y in (np.nextafter(1.0 / x, 0), 1.0 / x, np.nextafter(1.0 / x, 9))
              if _off(y, x) <= bound]
        assert len(ys) == 2
        X = int(np.ldexp(x, 53 - np.frexp(x)[1]))           # 53 bits
        # midpoints M (odd, 54 bits): random ones, and those that put X M next to a double, by
        # solving odd(X) M = j mod 2^54
        inv = pow(X // (X & -X), -1, 1 << 54)
        Ms = [int(k) * 2 + 1 for k in rng.integers(1 << 52, 1 << 53, 2000)]
        Ms += [M for M in (inv * j % (1 << 54) for j in range(-4001, 4002, 2)) if M >> 53]
        a = []
        for M in Ms:
            p = X * M
            sh = p.bit_length() - 53
            a += [float((p >> sh) + d) for d in (-1, 0, 1, 2)]
        a = np.array(a)
        for y in ys:
            got = np.empty_like(a)
            full = np.full_like(a, x), np.full_like(a, y)
            lib.quotients(*[v.ctypes.data_as(ctypes.c_void_p) for v in (a, *full)],
                          ctypes.c_int(len(a)), got.ctypes.data_as(ctypes.c_void_p))
            assert np.array_equal(got, a / x)
            tried += len(a)
    assert tried > 100000


@pytest.mark.parametrize("hi", [100, 400])
def test_plummer_terms(lib, hi):
    """The dwarf sampler's M / sqrt(r^2 + a^2), 1 / sqrt(x^5) (x^5 up to 2^400) and r / a."""
    rng = np.random.default_rng(hi)
    n = 500_000
    s = _random(rng, n, -100 if hi == 100 else 0, hi)
    m, x, a = _random(rng, n, -20, 20), _random(rng, n, -60, 45), _random(rng, n, -49, 49)
    x[:100] = 0.0
    x *= rng.choice([-1.0, 1.0], n)
    out = np.empty((n, 3))
    lib.plummer(*[v.ctypes.data_as(ctypes.c_void_p) for v in (s, m, x, a)], ctypes.c_int(n),
                out.ctypes.data_as(ctypes.c_void_p))
    want = np.stack([m / np.sqrt(s), 1.0 / np.sqrt(s), np.abs(x / a)], 1)
    out[:, 2] = np.abs(out[:, 2])           # the sign of a zero quotient is not kept
    ok = ~_near_ones(s)[:, None] & ~np.stack([np.zeros(n, bool)] * 2 + [_near_ones(a)], 1)
    assert np.array_equal(out.view(np.uint64)[ok], want.view(np.uint64)[ok])


def test_ranges(lib):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -701, 2.0 ** -700, 2.0 ** 699,
                  2.0 ** 700, -2.0 ** 699, 2.0 ** -101, 2.0 ** -100, 2.0 ** 99, 2.0 ** 100, -1.0])
    out = np.empty(len(x), np.int32)
    lib.ranges(x.ctypes.data_as(ctypes.c_void_p), ctypes.c_int(len(x)),
               out.ctypes.data_as(ctypes.c_void_p))
    ax = np.abs(x)
    with np.errstate(invalid="ignore"):
        want = ((ax >= 2.0 ** -700) & (ax < 2.0 ** 700)).astype(int) | \
               (((x >= 2.0 ** -100) & (x < 2.0 ** 100)).astype(int) << 1)
    assert (out & 3).tolist() == want.tolist() and (out >> 3 & 1).tolist() == (x == 0.0).tolist()
    x = np.array([2.0 - 2.0 ** -52, 2.0 - 2.0 ** -20, 2.0 - 2.0 ** -19, 1.0, 4.0 - 2.0 ** -51])
    out = np.empty(len(x), np.int32)
    lib.ranges(x.ctypes.data_as(ctypes.c_void_p), ctypes.c_int(len(x)),
               out.ctypes.data_as(ctypes.c_void_p))
    assert (out >> 2 & 1).tolist() == [1, 1, 0, 0, 1]
