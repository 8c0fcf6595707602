"""The FP64 operations that the kernels form in integers give the bits of the FP64 instructions in
whose place they stand: random operands, both sides of every range they are taken on, extreme and
sparse mantissas, ties, zeros, subnormals, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RCP, SQRT, MUL, FLOOR, INT, WIDEN, NARROW = range(7)
SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2e-308, -2.2e-308, 2.0 ** -1022,
                    np.finfo(float).max, -np.finfo(float).max])


def _floats(exponents, mantissas, signs=(0, 1)):
    e, m, s = (np.asarray(v, np.uint64) for v in (exponents, mantissas, signs))
    bits = (s[:, None, None] << np.uint64(63)) | (e[None, :, None] << np.uint64(52)) | m[None, None, :]
    return bits.reshape(-1).view(np.float64)


def _mantissas(rng, n):
    one = np.uint64(1)
    top = np.uint64((1 << 52) - 1)
    single = one << np.arange(52, dtype=np.uint64)
    near = np.arange(64, dtype=np.uint64)
    return np.unique(np.concatenate([single, top - single, near, top - near, rng.integers(0, 1 << 52, n, np.uint64)]))


def _same(which, a, b=None):
    from acum3_periodic_gb300 import native
    got, want = native.selftest_arith(which, a, b)
    g, w = got.view(np.int64), want.view(np.int64)
    bad = np.flatnonzero((g != w) & ~(np.isnan(got) & np.isnan(want)))
    assert bad.size == 0, (which, bad.size, a[bad[0]].hex(), (b if b is not None else a)[bad[0]].hex(),
                           got[bad[0]].hex(), want[bad[0]].hex())


def _edges(lo, hi):
    """Exponents around lo and hi (the ends of an operation's range as powers of two), and far off."""
    e = {1, 2, 500, 1023, 1024, 1500, 2045, 2046}
    for k in (lo, hi):
        e |= {1023 + k + d for d in (-2, -1, 0, 1, 2)}
    return sorted(x for x in e if 0 <= x <= 2046)


@pytest.mark.parametrize("which,lo,hi", [(RCP, -1000, 998), (SQRT, -900, 1000), (MUL, -255, 257), (FLOOR, 0, 30),
                                         (NARROW, -126, 127), (WIDEN, -126, 128)])
def test_ranges_and_mantissas(which, lo, hi):
    rng = np.random.default_rng(which)
    a = _floats(_edges(lo, hi), _mantissas(rng, 2000))
    a = np.concatenate([a, SPECIAL])
    if which == MUL:
        _same(which, a, rng.permutation(a))
        s = np.concatenate([SPECIAL, [1.0, -1.5, 2.0 ** -255, 2.0 ** -256, 2.0 ** 256, 2.0 ** 257]])
        _same(which, np.repeat(s, s.size), np.tile(s, s.size))
    else:
        _same(which, a)


@pytest.mark.parametrize("which", [RCP, SQRT, MUL])
def test_random_operands(which):
    rng = np.random.default_rng(10 + which)
    n = 1 << 23
    a = (rng.integers(0, 1 << 52, n, np.uint64) | (rng.integers(1000, 1040, n).astype(np.uint64) << np.uint64(52))).view(np.float64)
    b = rng.permutation(a) * np.where(rng.random(n) < 0.5, -1.0, 1.0)
    _same(which, a, b if which == MUL else None)


def test_product_ties():
    """Products of two odd 27-bit integers (54 bits: half a unit above a 53-bit value) and of 26
    and 27 bits (exact); both parities of the value below."""
    rng = np.random.default_rng(20)
    odd = lambda bits, n: (rng.integers(1 << (bits - 1), 1 << bits, n) | 1).astype(np.float64)  # noqa: E731
    for k in (26, 27):
        _same(MUL, odd(27, 1 << 20), odd(k, 1 << 20) * 2.0 ** -30)


def test_squares_and_their_neighbours():
    """Roots that are exact, and the values beside them."""
    rng = np.random.default_rng(21)
    r = rng.integers(1, 1 << 26, 1 << 18).astype(np.float64)
    q = np.concatenate([r * r, np.nextafter(r * r, 0.0), np.nextafter(r * r, np.inf)])
    _same(SQRT, np.concatenate([q, 2.0 * q]))


def test_integers():
    k = 2.0 ** np.arange(0, 32)
    n = np.concatenate([k, k - 1, k + 1, np.random.default_rng(22).integers(-2 ** 31, 2 ** 31, 1 << 18).astype(float)])
    n = np.concatenate([n, -n])
    n = n[(n >= -2.0 ** 31) & (n < 2.0 ** 31)]
    _same(INT, n)
    _same(FLOOR, np.concatenate([n, np.nextafter(n, -np.inf), np.nextafter(n, np.inf), n + 0.5]))


def test_float_rounding():
    """Doubles half way between two floats and beside it, of either parity, and floats themselves."""
    rng = np.random.default_rng(23)
    m = rng.integers(1 << 23, 1 << 24, 1 << 18).astype(np.float64)
    x = np.concatenate([m, m + 0.5, np.nextafter(m + 0.5, 0.0), np.nextafter(m + 0.5, np.inf)])
    for e in (-149, -130, -23, 0, 103, 104):
        _same(NARROW, x * 2.0 ** e)
        _same(NARROW, -x * 2.0 ** e)
    _same(WIDEN, (m * 2.0 ** -20).astype(np.float32).astype(np.float64))
