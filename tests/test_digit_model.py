"""A NumPy model of the digit products behind the FP64 chi0 (molgw_b200/csrc/digit_gemm.cu):
rows scaled to their largest entry, rounded to 55 bits, cut into seven balanced base-256
digits, digit products with i + j <= 9 summed exactly.  It pins what the kernel claims: the
digits are int8 and rebuild the integer, the INT32 sums of a chunk cannot overflow, and the
result is at least as close to an extended-precision sum as an FP64 sum is, whatever the range of
the energy differences and of the entries."""
import numpy as np
import pytest

NS, BITS, CHUNK = 7, 55, 16384


def exponents(x):
    m, e = np.frexp(np.abs(x).max(axis=1))
    return np.maximum(np.where(m > 0.996, e + 1, e), -960)


def digits(x):
    e = exponents(x)
    big = np.rint(np.ldexp(x, (BITS - e)[:, None])).astype(np.int64)
    bias = np.int64(sum(128 << (8 * k) for k in range(NS - 1)))
    y = (big + bias) ^ bias
    d = np.stack([((y >> (8 * (NS - i))) & 255).astype(np.uint8).view(np.int8) for i in range(1, NS)]
                 + [(y & 255).astype(np.uint8).view(np.int8)])
    top = (big + bias) >> (8 * (NS - 1))
    assert np.all(np.abs(top) <= 127)
    return d.astype(np.int64), e, big


def digit_product(a, b):
    da, ea, _ = digits(a)
    db, eb, _ = digits(b)
    out = np.zeros((a.shape[0], b.shape[0]))
    for k in range(0, a.shape[1], CHUNK):
        lo, hi = np.zeros(out.shape, np.int64), np.zeros(out.shape, np.int64)
        for d in range(2, NS + 3):
            lev = sum(da[i - 1][:, k:k + CHUNK] @ db[d - i - 1][:, k:k + CHUNK].T
                      for i in range(max(1, d - NS), min(NS, d - 1) + 1))
            assert np.abs(lev).max() < 2 ** 31
            if d <= NS - 2:
                hi = hi * 256 + lev
            else:
                lo = lo * 256 + lev
        out += lo.astype(float)
        out += hi.astype(float) * 2.0 ** 32
    if a is b:                                   # squares of digit 5, of the first level left out
        out += np.diag((da[4] ** 2).sum(axis=1) * 2.0 ** -8)
    return np.ldexp(out, ea[:, None] + eb[None, :] + 8 * (NS - 2) - 2 * BITS)


def test_digits_rebuild_the_integer_and_fit_int8():
    rng = np.random.default_rng(0)
    x = rng.standard_normal((9, 400)) * 10.0 ** rng.uniform(-200, 200, (9, 1))
    x[0, :4] = [0.0, 1.0, -1.0, 0.996]           # row maximum at the edge of the leading digit
    x[0, 4:] = 0.0
    x[1] = 0.0
    x[2] *= 1e-280
    d, e, big = digits(x)
    assert np.array_equal(sum(d[i - 1] << (8 * (NS - i)) for i in range(1, NS + 1)), big)
    full = np.ldexp(big.astype(float), (e - BITS)[:, None])
    assert np.all(np.abs(full - x).max(axis=1) <= np.ldexp(1.0, e - BITS - 1) * 1.0001 + 0.0)


def test_largest_levels_stay_inside_int32():
    # every digit at its extreme: 7 products of level 8 over one chunk
    assert 7 * 128 * 128 * CHUNK < 2 ** 31


@pytest.mark.parametrize("k", [512, 1890, 4347, 25000])
@pytest.mark.parametrize("spread", [0.0, 3.0, -1.0])
@pytest.mark.parametrize("gaps,rising", [(0.0, False), (3.0, False), (3.0, True)])
def test_error_is_no_larger_than_an_fp64_sum(k, spread, gaps, rising):
    """2-norm of the error, relative to sqrt(C_pp C_qq), against an extended-precision sum;
    ``spread``: decades over which the entries of a row vary (0: the normal draw; -1: three large
    ones in every row and the rest 1e-4 of them), ``gaps``: decades of the energy differences,
    ``rising``: amplitudes that grow as their roots."""
    rng = np.random.default_rng(k)
    m = rng.standard_normal((24, k)) * 10.0 ** (-max(spread, 0.0) * rng.random((24, k)))
    if spread < 0.0:
        m *= 1.0e-4
        m[np.arange(24)[:, None], rng.integers(0, k, (24, 3))] = 1.0
    de = 10.0 ** (-1.0 + gaps * rng.random(k)) if gaps else rng.uniform(0.3, 2.5, k)
    if rising:
        m *= np.sqrt(de)
    d = 4.0 / de
    ref = np.zeros((24, 24), np.longdouble)
    for c in range(0, k, 500):
        ref += ((m[:, c:c + 500].astype(np.longdouble) * d[c:c + 500])[:, None, :] *
                m[None, :, c:c + 500].astype(np.longdouble)).sum(axis=2)
    a = m * d
    seq = np.zeros((24, 24))
    for t in range(0, k, 4):                      # four transitions per DMMA step
        seq += a[:, t:t + 4] @ m[:, t:t + 4].T
    s = m * np.sqrt(d)
    scale = np.sqrt(np.outer(np.diag(ref), np.diag(ref)))
    err = [float(np.linalg.norm(((c - ref) / scale).astype(float))) for c in (digit_product(s, s), seq)]
    assert err[0] <= err[1], err


@pytest.mark.parametrize("ns", [4, 6])
def test_squares_of_the_middle_digit_on_the_diagonal(ns):
    """An even number of digits: the level left out first holds the squares of digit ns/2 + 1 on the
    diagonal, whose mean is not zero; with their sum added the diagonal is as close as the rest."""
    rng = np.random.default_rng(ns)
    x = rng.standard_normal((16, 3000))
    bits = 8 * ns - 1
    e = exponents(x)
    big = np.rint(np.ldexp(x, (bits - e)[:, None])).astype(np.int64)
    bias = np.int64(sum(128 << (8 * k) for k in range(ns - 1)))
    y = (big + bias) ^ bias
    d = [((y >> (8 * (ns - i))) & 255).astype(np.uint8).view(np.int8).astype(np.int64) for i in range(1, ns + 1)]
    out = sum((d[i - 1] @ d[j - 1].T).astype(np.longdouble) * np.longdouble(2.0) ** (8 * (2 * ns - i - j))
              for i in range(1, ns + 1) for j in range(1, ns + 1) if i + j <= ns + 1)
    ref = big.astype(np.longdouble) @ big.T.astype(np.longdouble)
    norm = np.sqrt(np.outer(np.diag(ref), np.diag(ref)))
    off = ~np.eye(16, dtype=bool)
    rest = np.sqrt(np.mean(((out - ref) / norm)[off] ** 2))
    plain = np.diag((out - ref) / norm)
    squares = (d[ns // 2] ** 2).sum(axis=1).astype(np.longdouble) * np.longdouble(2.0) ** (8 * (ns - 2))
    fixed = np.diag((out + np.diag(squares) - ref) / norm)
    assert np.abs(plain).min() > 10 * rest
    assert np.sqrt(np.mean(fixed ** 2)) < 3 * rest
