"""The shared-seed roots, reciprocals and quotients of the force terms
(fn_rounded.cuh) against the host's IEEE operations, every bit: the operands
whose exact results lie closest to the middle of two doubles, the edges of the
range they are used in, and random ones."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HERE = os.path.join(ROOT, "tests", "rounded")
HEADER = os.path.join(ROOT, "fibrenet_b200", "csrc", "fn_rounded.cuh")
OP_ROOT, OP_INVERSE_ROOT, OP_PRODUCT_INVERSE, OP_SQUARE_INVERSE, OP_QUOTIENT, OP_QUOTIENT_ANY, \
    OP_SQUARE_QUOTIENT = range(7)

# 2^106 - k = product of the primes, k = 1 .. 16
FACTORS = {
    1: [3, 107, 6361, 69431, 20394401, 28059810762433],
    2: [2, 7, 7, 31, 71, 127, 151, 337, 29191, 106681, 122921, 152041],
    3: [2327027, 34864072662073401681969743],
    4: [2, 2, 3, 5, 17, 53, 157, 1613, 2731, 8191, 858001, 308761441],
    5: [19, 29, 147240723075511219048618884109],
    6: [2, 67, 577, 61845503, 16966443015568478977],
    7: [3, 3, 3, 223, 449, 30009901652533386930372133],
    8: [2, 2, 2, 2550183799, 3976656429941438590393],
    9: [5, 7, 11, 1187, 2203, 5741, 712176643, 19709623201],
    10: [2, 3, 13, 782489, 9763970147, 136138278236071],
    11: [83, 5417, 105615816899, 1708494755208277],
    12: [2, 2, 541, 6719, 517189, 10788681283839114323],
    13: [3, 23, 79, 11465977, 1298052602016345651713],
    14: [2, 5, 5, 311, 5217340090971490784295112871],
    15: [1233003839411, 65798366413329190859],
    16: [2, 2, 2, 2, 3, 3, 7, 103, 307, 2143, 2857, 6529, 11119, 43691, 131071],
}


def hard_reciprocals():
    """Mantissas b in [2^52, 2^53) with b m = 2^106 - k: m, a whole number of
    54 bits, is the middle of two doubles and 1/b lies k 2^-106 of it above."""
    out = set()
    for k, primes in FACTORS.items():
        divisors = {1}
        product = 1
        for p in primes:
            product *= p
            divisors |= {d * p for d in divisors if d * p < 1 << 53}
        assert product == (1 << 106) - k
        out |= {d for d in divisors if d >= 1 << 52}
    return np.ldexp(np.array(sorted(out), np.float64), -52)


def roots_mod(c, n):
    """All x in [0, 2^n) with x^2 = c mod 2^n, c = 1 mod 8."""
    xs, m = {1, 3, 5, 7}, 3
    while m < n:
        m += 1
        xs = {t % 2**m for x in xs for t in (x, x + 2 ** (m - 1)) if (t * t - c) % 2**m == 0}
    return xs


def hard_roots():
    """Doubles d whose root lies next to the middle m / 2^53 of two doubles:
    d 2^106 - m^2 = k for small k, in two binades."""
    out = set()
    for k in range(-4089, 4097, 8):  # odd m: k = -m^2 = 7 mod 8
        for n, lo in ((54, 106), (55, 107)):
            for r in roots_mod(-k % 2**n, n):
                for m in {r, r + 2**n}:
                    q = m * m + k
                    if 2**53 <= m < 2**54 and 2**lo <= m * m < 2 ** (lo + 1) and q % 2**n == 0 and 2**52 <= q >> n < 2**53:
                        out.add(float(q >> n) * (2.0**-52 if n == 54 else 2.0**-51))
    return np.array(sorted(out))


def around(x, ulps):
    """x and its neighbours."""
    bits = np.asarray(x, np.float64).view(np.int64)
    return np.concatenate([(bits + k).view(np.float64) for k in range(-ulps, ulps + 1)])


def binades(x, powers):
    return np.concatenate([np.ldexp(x, p) for p in powers])


def randoms(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    return np.ldexp(1.0 + rng.random(n), rng.integers(lo, hi, n))


EDGES = np.concatenate([around(np.ldexp(1.0, [-200, -199, -2, -1, 0, 1, 2, 199, 200]), 3), [2.0**53 - 1.0]])
SPECIAL = np.array([0.0, -0.0, 5e-324, 2.0**-1022, 2.0**-540, 2.0**600, np.finfo(float).max, np.inf, np.nan, -1.0])


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from fibrenet_b200 import build
    lib = str(tmp_path_factory.mktemp("rounded") / "librounded.so")
    out = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-shared", "-o", lib, os.path.join(HERE, "harness.cu")],
                         capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-3000:]
    f = C.CDLL(lib).fr_run
    f.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_longlong]

    def call(op, a, b=None):
        a = np.ascontiguousarray(a, np.float64)
        b = np.ones_like(a) if b is None else np.ascontiguousarray(b, np.float64)
        out = np.empty_like(a)
        assert f(op, a.ctypes.data, b.ctypes.data, out.ctypes.data, a.size) == 0
        return out

    return call


def same_bits(got, want, *operands):
    bad = np.flatnonzero((got.view(np.int64) != want.view(np.int64)) & ~(np.isnan(got) & np.isnan(want)))
    assert bad.size == 0, f"{bad.size} of {got.size} differ, e.g. " + str(
        [float(v[bad[0]]).hex() for v in (*operands, got, want)])


def inverse(x):
    with np.errstate(divide="ignore", invalid="ignore"):
        return np.where(x != 0.0, 1.0 / x, 0.0)


def root_operands():
    """Arguments of a root whose root, or whose root's reciprocal, is hard to
    round; the edges of the range; random ones."""
    b = hard_reciprocals()
    near = [around(np.ldexp(b * b, p), 2) for p in (-200, -3, -2, -1, 0, 1, 2, 3, 196)]
    return np.concatenate([binades(hard_roots(), (-198, -2, 0, 2, 196)), *near, EDGES, SPECIAL,
                           randoms(4_000_000, -200, 200, 1), randoms(4_000_000, -4, 4, 2)])


def test_lists_of_hard_operands():
    assert len(hard_reciprocals()) > 250 and len(hard_roots()) > 1000


def test_root(run):
    d = root_operands()
    with np.errstate(invalid="ignore"):
        same_bits(run(OP_ROOT, d), np.sqrt(d), d)


def test_inverse_of_a_root(run):
    d = root_operands()
    with np.errstate(invalid="ignore"):
        same_bits(run(OP_INVERSE_ROOT, d), inverse(np.sqrt(d)), d)


def test_inverse_of_a_square(run):
    b = hard_reciprocals()
    edges = EDGES[(EDGES >= 2.0**-200) & (EDGES < 2.0**200)]
    d = np.concatenate([binades(b, range(-200, 200)), edges, randoms(4_000_000, -200, 200, 3)])
    same_bits(run(OP_SQUARE_INVERSE, d), 1.0 / d, d)


def test_inverse_of_a_product(run):
    """The reciprocal of a product of two roots from the roots' reciprocals."""
    hard = hard_reciprocals()
    rng = np.random.default_rng(4)
    a = np.ldexp(1.0 + rng.random(4_000_000), rng.integers(-4, 5, 4_000_000))
    la = np.sqrt(a)
    lb = hard[rng.integers(0, hard.size, a.size)] / la
    b = lb * lb
    ones = binades(hard, (-1, 0, 1))
    a = np.concatenate([a, np.ones(ones.size), randoms(2_000_000, -90, 90, 5)])
    b = np.concatenate([b, ones * ones, randoms(2_000_000, -90, 90, 6)])
    product = np.sqrt(a) * np.sqrt(b)
    mantissa = np.frexp(product)[0] * 2.0
    assert np.isin(mantissa, hard).sum() > 100_000
    same_bits(run(OP_PRODUCT_INVERSE, a, b), 1.0 / product, a, b)


def numerators(b, k):
    """The mantissas a for which a/b lies next to the middle m of two doubles:
    a 2^54 - b m = k or a 2^53 - b m = k, b and k odd (an even b keeps its
    quotients twice as far from any middle)."""
    for p in (53, 54) if b % 2 else ():
        m = -k * pow(b, -1, 1 << p) % (1 << p)
        m += (1 << 53) if m < 1 << 53 and p == 53 else 0
        a = (b * m + k) >> p
        if (1 << 53) <= m < (1 << 54) and (1 << 52) <= a < (1 << 53):
            yield a


def hard_quotients(n, seed):
    rng = np.random.default_rng(seed)
    out = []
    while len(out) < n:
        b = int(rng.integers(1 << 52, 1 << 53)) | 1
        out += [(a, b) for a in numerators(b, int(rng.integers(-8, 8)) * 2 + 1)]
    for b in np.ldexp(hard_reciprocals(), 52).astype(np.int64):
        out += [(a, int(b)) for k in range(-15, 16, 2) for a in numerators(int(b), k)]
    a, b = np.array(out, np.float64).T
    return np.ldexp(a, -52), np.ldexp(b, -52)


@pytest.mark.parametrize("op", [OP_QUOTIENT, OP_SQUARE_QUOTIENT])
def test_quotient(run, op):
    ha, hb = hard_quotients(60_000, 7)
    rb = hard_reciprocals()
    rng = np.random.default_rng(8)
    a = np.concatenate([ha, -ha, 1.0 + rng.random(rb.size * 50), randoms(4_000_000, -200, 200, 9)])
    b = np.concatenate([hb, hb, np.repeat(rb, 50), randoms(4_000_000, -200, 200, 10)])
    same_bits(run(op, a, b), a / b, a, b)


def test_quotient_of_any_numerator(run):
    """Zeros, infinities, NaN and numerators at the ends of the range of doubles
    and of the fast sequence, over divisors as roots are."""
    rng = np.random.default_rng(12)
    tiny = np.array([5e-324, 3e-320, 2.0**-1022, 2.0**-970, np.finfo(float).max, 0.0, np.inf])
    edges = around(np.ldexp(1.0, [-401, -400, -399, 399, 400, 401]), 2)
    a = np.concatenate([tiny, edges, randoms(20_000, -1070, 1023, 13)])
    a = np.concatenate([a, -a, [np.nan]])
    b = np.concatenate([1.0 + rng.random(64), np.ldexp(1.0 + rng.random(64), rng.integers(-537, 511, 64)),
                        hard_reciprocals()[::8], np.ldexp(1.0, [-537, -200, -1, 0, 1, 511])])
    a, b = (np.ascontiguousarray(v).ravel() for v in np.meshgrid(a, b))
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        same_bits(run(OP_QUOTIENT_ANY, a, b), a / b, a, b)
