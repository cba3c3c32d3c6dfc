"""The fixed-point digit products of the complex128 kernels, restated in numpy.

fx.cuh holds a matrix as 64-bit integers at one exponent, |v| <= 2^62, and cuts
an integer into seven digits q_s in [-128, 127] with |q_0| <= 64.  The tensor
core sums the digit products of a level s + t <= 7 over 64 complex columns (128
real terms) in FP32.  Checked here on random and on extreme operands:

  * the digits reproduce the integer to half a unit of its eighth byte;
  * every level sum stays below 2^24 (FP32 holds it), levels 0 .. 2 within 2^22
    (the kernels turn those into integers with one addition), whatever the
    digits;
  * the product of the kept levels is no further from the exact one than FP64
    matrix products are, for general matrices and for the E P products of a
    propagation.
"""
import numpy as np
import pytest

S, LEVELS, TERMS = 7, 8, 128


def digits(v):
    u = v.astype(np.uint64) + np.uint64(0x8080808080808080)
    return [((u >> np.uint64(8 * (7 - s))) & np.uint64(255)).astype(np.int64) - 128 for s in range(S)]


def fixed(x):
    m = max(np.abs(x.real).max(), np.abs(x.imag).max())
    e = int(np.floor(np.log2(m))) + 1
    return [np.rint(np.ldexp(p.astype(np.longdouble), 62 - e)).astype(np.int64) for p in (x.real, x.imag)], e


def product(A, B):
    """The kept levels of A B, in long double."""
    (ar, ai), ea = fixed(A)
    (br, bi), eb = fixed(B)
    Aq = [np.block([[r, -i], [i, r]]).astype(np.float64) for r, i in zip(digits(ar), digits(ai))]
    Bq = [np.vstack([r, i]).astype(np.float64) for r, i in zip(digits(br), digits(bi))]
    T = np.zeros((2 * A.shape[0], B.shape[1]), dtype=np.longdouble)
    for L in range(LEVELS):
        D = sum(Aq[s] @ Bq[L - s] for s in range(S) if 0 <= L - s < S)
        T += D.astype(np.longdouble) * np.longdouble(2.0) ** (-8 * L + ea + eb - 12)
    n = A.shape[0]
    return T[:n], T[n:]


def test_digits_reproduce_the_integer():
    rng = np.random.default_rng(0)
    edge = [0, 1, -1, 127, 128, -128, -129, 2 ** 62, -2 ** 62, 2 ** 62 - 1, 1 - 2 ** 62, 2 ** 61, 0x7F7F7F7F7F7F7F]
    v = np.concatenate([np.array(edge, dtype=np.int64), rng.integers(-2 ** 62, 2 ** 62, 100000)])
    q = digits(v)
    assert np.abs(q[0]).max() <= 64
    assert all(x.min() >= -128 and x.max() <= 127 for x in q[1:])
    back = sum(x.astype(object) * 2 ** (8 * (7 - s)) for s, x in enumerate(q))
    assert max(abs(int(b) - int(x)) for b, x in zip(back, v)) <= 128


def test_level_sums_stay_exact():
    """The largest possible level sums of 128 terms (4 stages of 32)."""
    top = [64] + [128] * (S - 1)
    for L in range(LEVELS):
        worst = TERMS * sum(top[s] * top[L - s] for s in range(S) if 0 <= L - s < S)
        assert worst < 2 ** 24
        if L <= 2:
            assert worst <= 2 ** 22


@pytest.mark.parametrize("d", [16, 65, 128])
@pytest.mark.parametrize("kind", ["hermitian", "near_identity", "unitary"])
def test_products_are_no_further_off_than_fp64(d, kind):
    rng = np.random.default_rng(d)
    a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
    X = (a + a.conj().T) / (4 * np.sqrt(d))
    U = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))[0]
    A, B = {"hermitian": (X, X), "near_identity": (-0.1j * X, U), "unitary": (U, U.conj().T @ X)}[kind]
    L = np.longdouble
    re = A.real.astype(L) @ B.real.astype(L) - A.imag.astype(L) @ B.imag.astype(L)
    im = A.real.astype(L) @ B.imag.astype(L) + A.imag.astype(L) @ B.real.astype(L)
    tr, ti = product(A, B)
    C = A @ B

    def off(r, i):
        return float(np.sqrt(((r - re) ** 2).sum() + ((i - im) ** 2).sum()))

    assert off(tr, ti) <= off(C.real, C.imag)
