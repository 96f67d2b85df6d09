"""The FP64 exchange on int8 products (i8_digits.cuh, k_xform_i8.cu, k_exchange_i8.cu), restated in numpy and run on the
fitted integrals of a water dimer.  Values become seven balanced byte digits, v = sum_s d_s 256^(6-s) with one
exponent per B^Q, per orbital and per row of X^T; of the digit products those with s + t < 8 are kept, 34 of 49, each
an exact integer.  Functions of very unequal size get row scales, powers of two that make every row's largest
element of B about 1.

Each operand is rounded at 2^-55 of its largest element, below the 2^-53 of an FP64 value.  The bound is what an FP64
sum of the n + n_aux n_c = 2,368 terms may leave, 2,368 x 2^-53 = 2.6e-13 of the sum of the terms' magnitudes, which
is at most sqrt(K_mm K_nn); the reference is formed in extended precision.  Multiplying the functions by powers of two
changes nothing in exact arithmetic, so the bound holds for any spread of them."""
import numpy as np
import pytest

import rijk_oracle as O
from nopt_b200 import ints
from nopt_b200.molecules import water_cluster


def exponent(top):
    """value_exponent: top / 2^x <= 127.49 2^48."""
    f, e = np.frexp(top)
    return np.where(top > 0, np.where(f > 0.995, e + 1, e) - 55, 0).astype(int)


def digits(x, ex):
    """digits16: balanced bytes, the leading one first."""
    v = np.rint(np.ldexp(x, -ex)).astype(np.int64)
    out = []
    for _ in range(7):
        d = ((v + 128) & 255) - 128
        out.append(d)
        v = (v - d) >> 8
    assert not v.any()
    return out[::-1]


def products(a, b):
    """34 products of digits, joined as the kernels do: sum_{g<8} G_g 256^(12-g)."""
    G = [0] * 8
    count = 0
    for s in range(7):
        for t in range(min(7, 8 - s)):
            G[s + t] = G[s + t] + a[s].astype(float) @ b[t].T.astype(float)
            count += 1
    assert count == 34
    assert max(np.max(np.abs(g)) for g in G) < 2 ** 31 - 1
    hi, lo = ([int(256 ** (3 - g)) * G[h + g].astype(np.int64) for g in range(4)] for h in (0, 4))
    return np.ldexp(sum(lo).astype(float) * 2.0 ** -32 + sum(hi).astype(float), 72)


def row_scales(B):
    """k_balance, k_spread: exponents e with max_{Q, nu} 2^-(e_mu + e_nu) |B| about 1; none if that holds to a factor 11 (2^(2 x 1.75))."""
    with np.errstate(divide="ignore"):
        L = np.log2(np.max(np.abs(B), axis=0))
    e = np.zeros(len(L))
    for step in range(8):
        e = 0.5 * (e + np.max(L - e[None, :], axis=1))
        if step == 0 and np.ptp(e) <= 1.75:
            return np.zeros(len(L), int)
    return np.rint(e).astype(int)


def exchange(B, C):
    naux, n, _ = B.shape
    e = row_scales(B)
    Bs, Cs = np.ldexp(B, -(e[:, None] + e[None, :])), np.ldexp(C, e[None, :])
    xc = exponent(np.max(np.abs(Cs), axis=1))
    dc = digits(Cs, xc[:, None])
    X = np.empty((n, naux, len(C)))
    for q in range(naux):
        xq = exponent(np.max(np.abs(Bs[q])))
        X[:, q] = np.ldexp(products(digits(Bs[q], xq), dc), xq + xc[None, :] + e[:, None])
    X = X.reshape(n, -1)
    xr = exponent(np.max(np.abs(X), axis=1))
    d = digits(X, xr[:, None])
    return np.ldexp(products(d, d), xr[:, None] + xr[None, :])


@pytest.fixture(scope="module")
def dimer():
    si = ints.SystemIntegrals(water_cluster((1, 1, 2), seed=0), "cc-pvdz", "cc-pvdz-jkfit")
    B = (O.s05_calc(si.V)[0] @ O.unpack_3c(si.I3, si.n).T).reshape(si.naux, si.n, si.n)
    B = 0.5 * (B + B.transpose(0, 2, 1))
    C = np.linalg.qr(np.random.default_rng(0).normal(size=(si.n, si.n)))[0].T[:si.nocc]
    X = np.einsum("qnm,im->nqi", B.astype(np.longdouble), C.astype(np.longdouble)).reshape(si.n, -1)
    return B, C, X @ X.T


@pytest.mark.parametrize("spread", [0, 3, 12, 60])
def test_exchange_from_digits(dimer, spread):
    B, C, K = dimer
    n, terms = len(K), B.shape[1] + B.shape[0] * len(C)
    s = -np.random.default_rng(spread).integers(0, spread + 1, n)
    assert np.any(row_scales(np.ldexp(B, s[:, None] + s[None, :]))) == (spread > 0)
    got = exchange(np.ldexp(B, s[:, None] + s[None, :]), np.ldexp(C, -s[None, :]))
    got = np.ldexp(got, -(s[:, None] + s[None, :]))
    d = np.sqrt(np.diag(K))
    assert np.max(np.abs(got - K) / np.outer(d, d)) <= terms * 2.0 ** -53


def test_digits_hold_their_values(dimer):
    """Every value comes back to half a unit of the last digit, 2^-55 of the largest."""
    x = dimer[0][5]
    ex = exponent(np.max(np.abs(x)))
    d = digits(x, ex)
    back = sum(v.astype(np.longdouble) * np.longdouble(256) ** (6 - s) for s, v in enumerate(d))
    err = np.abs(back - np.ldexp(x.astype(np.longdouble), -ex))
    assert np.max(err) <= 0.5
    assert np.max(np.abs(x)) * 2.0 ** -55 >= np.ldexp(0.5, ex)
    assert all(v.min() >= -128 and v.max() <= 127 for v in d)
