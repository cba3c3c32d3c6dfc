"""complex128 results as close to exact ones as FP64 products are: propagators with
little mixing (nearly diagonal Hamiltonians, where sums bounded by 2 d terms would leave
most of an accumulator unused), large steps, and lossy ones whose size falls by ten
decades.

The exact propagator is formed in long double (113 or 64 bits); for the lossy ones, whose
eigenvalues lie off the real axis, from the contexts' own Chebyshev polynomial, since the
order does not resolve them to 2^-53.  Bars, relative to its Frobenius norm: a product of FP64 matrices is off
by a few units of 2^-53 per row, here 2e-16 (5 + sqrt(P)) for P steps, and 1e-16 P for
what rounds the same way at every step (J_0 in the recurrence).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def exact(H0, H1, u, dt):
    CL, L = np.clongdouble, np.longdouble
    d = H0.shape[0]
    U, eye = np.eye(d, dtype=CL), np.eye(d, dtype=CL)
    for j in range(u.shape[1]):
        A = (CL(-1j) * L(dt)) * (H0.astype(CL) + sum(CL(u[k, j]) * H1[k].astype(CL) for k in range(len(H1))))
        V = eye
        for n in range(20, 0, -1):
            V = eye + (A @ V) / L(n)
        U = V @ U
    return U


def chebyshev(H0, H1, u, dt, hn, M):
    """The product of the steps' polynomials of order M in long double, from the Bessel
    functions as the contexts have them (the C library's)."""
    import oracle
    CL, L = np.clongdouble, np.longdouble
    d = H0.shape[0]
    U, eye = np.eye(d, dtype=CL), np.eye(d, dtype=CL)
    J = oracle.bessel_coeffs(M, hn * dt).astype(CL)  # (-i)^k J_k
    for j in range(u.shape[1]):
        X = (H0.astype(CL) + sum(CL(u[k, j]) * H1[k].astype(CL) for k in range(len(H1)))) / L(hn)
        T0, T1 = eye, X
        V = J[0] * eye + L(2) * J[1] * X
        for k in range(2, M + 1):
            T0, T1 = T1, L(2) * (X @ T1) - T0
            V = V + L(2) * J[k] * T1
        U = V @ U
    return U


def hermitian(rng, d):
    a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
    return (a + a.conj().T) / (4 * np.sqrt(d))


def off(U, X):
    return float(np.sqrt((np.abs(U.astype(np.clongdouble) - X) ** 2).sum() / (np.abs(X) ** 2).sum()))


def bar(P):
    return 2e-16 * (5 + np.sqrt(P)) + 1e-16 * P


def solve(H0, H1, u, dt):
    import parament_gb300 as parament
    with parament.Parament("fp64") as ctx:
        ctx.set_hamiltonian(H0, *H1)
        return ctx.equiprop(dt, *u), ctx.hamiltonian_norm, ctx.last_iteration_cycles


@pytest.mark.parametrize("d,P", [(4, 60), (12, 60), (20, 40), (24, 40), (33, 24), (64, 6), (72, 4)])
@pytest.mark.parametrize("mixing", [0.01, 1.0])
@pytest.mark.parametrize("x", [0.05, 0.5, 0.95])
def test_little_mixing_and_large_steps(built_lib, d, P, mixing, x):
    rng = np.random.default_rng((d, P))
    H0 = np.diag(rng.uniform(-1, 1, d)) + mixing * hermitian(rng, d)
    H1 = np.stack([np.diag(0.3 * rng.uniform(-1, 1, d)) + mixing * hermitian(rng, d)])
    u = rng.uniform(-1, 1, (1, P))
    dt = x / sum(np.abs(m).sum(0).max() for m in (H0, *H1))
    assert off(solve(H0, H1, u, dt)[0], exact(H0, H1, u, dt)) < bar(P)


# Two problems miss the bar: their loss alone takes x above 1 (to 1.005 and 4.6), where the
# bar's premise (x below 1) fails.  (14, 80) is 1.8e-12 off in the FP64 step kernel,
# (70, 6) 4.2e-13 in the fixed point and 3.6e-13 in the FP64 oracle.
ILL = pytest.mark.xfail(reason="strongly lossy steps above x = 1: the recurrence's own conditioning")
DECAY = [(d, P, k) if (d, P, k) not in [(14, 80, 10), (70, 6, 10)] else pytest.param(d, P, k, marks=ILL)
         for d, P in [(2, 300), (8, 120), (14, 80), (20, 160), (36, 24), (70, 6)] for k in (3, 10)]


@pytest.mark.parametrize("d,P,decades", DECAY)
def test_decay(built_lib, d, P, decades):
    """A uniform loss beside a Hermitian rest: the propagator's size falls by `decades`."""
    rng = np.random.default_rng((d, P, decades))
    H0, H1, u = hermitian(rng, d), hermitian(rng, d)[None], rng.uniform(-1, 1, (1, P))
    gamma = 1.0
    dt = decades * np.log(10.0) / gamma / P
    hn = sum(np.abs(m).sum(0).max() for m in (H0 - 1j * gamma * np.eye(d), *H1))
    scale = min(1.0, 0.9 / (hn * dt))  # x below 1: the Hermitian rest gives way
    H0, H1 = H0 * scale - 1j * gamma * np.eye(d), H1 * scale
    U, hn, M = solve(H0, H1, u, dt)
    assert off(U, chebyshev(H0, H1, u, dt, hn, M)) < 3 * bar(P)


@pytest.mark.parametrize("d,cycles,x", [(36, 3, 2.5), (36, 9, 30.0), (72, 3, 8.1), (72, 9, 55.0), (72, 13, 7.9)])
def test_two_large_steps(built_lib, d, cycles, x):
    """Two steps far beyond what the order resolves, against the oracle (the polynomial is
    no exponential)."""
    import oracle
    import parament_gb300 as parament
    rng = np.random.default_rng((d, cycles))
    H0, H1, u = hermitian(rng, d), hermitian(rng, d)[None], rng.uniform(-1, 1, (1, 2))
    hn = sum(np.abs(m).sum(0).max() for m in (H0, *H1))
    with parament.Parament("fp64") as ctx:
        ctx.set_hamiltonian(H0, *H1)
        ctx.set_iteration_cycles_manually(cycles)
        U = ctx.equiprop(x / hn, *u)
    Uo = oracle.equiprop(H0, H1, u, x / hn, M=cycles)[0]
    assert np.linalg.norm(U - Uo) / np.sqrt(d) < 2e-16 * (cycles + 10) * 2
