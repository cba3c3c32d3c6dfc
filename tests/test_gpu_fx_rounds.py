"""k_fx_gemm over several rounds of steps: chunks of more than one step, the last round
short of some of them (their products are carried over), the running product and the
tree, in each of its forms, with the orders and inputs that reach it.

Bars: complex128 4e-16 per step and 4e-15 (as in test_gpu_fx.py); plain complex64
1e-5 and 2e-8 per step (the grid of U_j's diagonal, 2^-25 coherent at worst); split
form 1e-6.
"""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
SMS = 152


def problem(precision, d, K, P, hermitian=True):
    rng = np.random.default_rng((d, K, P))

    def h():
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        if hermitian:
            a = a + a.conj().T
        return a / (4 * np.sqrt(d))

    H0, H1, u = h(), np.stack([h() for _ in range(K)]), rng.uniform(-1.0, 1.0, (K, P)) + 0j
    if precision == "fp32":
        H0, H1, u = (x.astype(np.complex64).astype(np.complex128) for x in (H0, H1, u))
    return H0, H1, u, float(sum(np.abs(m).sum(0).max() for m in (H0, *H1)))


def rounds(d, P):
    """(chunks, steps of the shorter chunks, longer ones), as make_plan cuts them."""
    tiles = ((d + 63) // 64) ** 2
    g = min(P, (16 * SMS + tiles - 1) // tiles)
    n = -(-P // -(-P // g))
    return n, P // n, P % n


def check(precision, form, H0, H1, u, dt, cycles=0):
    import parament_gb300 as parament
    P = u.shape[1]
    with parament.Parament(precision) as ctx:
        if form == "split":
            ctx.set_precision_mode("split")
        ctx.set_hamiltonian(H0, *H1)
        if cycles:
            ctx.set_iteration_cycles_manually(cycles)
        U, M = ctx.equiprop(dt, *u), ctx.last_iteration_cycles
    if form == "plain" and precision == "fp32":
        tiles = ((H0.shape[0] + 63) // 64) ** 2
        assert P * tiles * (H0.shape[0] * M - 420) >= 155000  # the line to these kernels
    Uo, Mo = oracle.equiprop(H0, H1, u, dt, single=precision == "fp32" and form == "plain",
                             M=cycles or (M if form == "split" else 0), nthreads=os.cpu_count())[:2]
    assert M == Mo
    bar = 4e-16 * P + 4e-15 if precision == "fp64" else 1e-6 if form == "split" else 1e-5 + 2e-8 * P
    assert np.linalg.norm(U - Uo) / np.linalg.norm(Uo) < bar
    return M


@pytest.mark.parametrize("precision,form,d,P,x", [
    ("fp32", "plain", 96, 1501, 0.1), ("fp32", "plain", 200, 320, 0.02), ("fp32", "plain", 260, 200, 0.3),
    ("fp32", "split", 80, 1300, 0.1), ("fp32", "split", 129, 601, 0.4), ("fp64", "plain", 72, 1301, 0.05),
    ("fp64", "plain", 129, 700, 0.02), ("fp64", "plain", 100, 1219, 1.3)])
def test_uneven_rounds(built_lib, precision, form, d, P, x):
    n, short, longer = rounds(d, P)
    assert short >= 2 and 0 < longer < n
    H0, H1, u, hn = problem(precision, d, 2, P)
    check(precision, form, H0, H1, u, x / hn)


@pytest.mark.parametrize("x,cycles", [(0.5, 0), (0.95, 0), (0.3, 9), (0.3, 11), (0.3, 13), (0.3, 15), (0.3, 21)])
def test_orders_of_the_plain_complex64_form(built_lib, x, cycles):
    H0, H1, u, hn = problem("fp32", 80, 2, 400)
    assert check("fp32", "plain", H0, H1, u, x / hn, cycles) >= 7


@pytest.mark.parametrize("form", ["plain", "split"])
def test_general_matrices_and_complex_controls(built_lib, form):
    H0, H1, u, hn = problem("fp32", 90, 18, 700, hermitian=False)
    u = (u + 1j * np.roll(u, 1, axis=1)).astype(np.complex64).astype(np.complex128) / 32
    check("fp32", form, H0, H1, u, 0.4 / hn)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_samples_that_are_not_finite(built_lib, bad):
    import parament_gb300 as parament
    H0, H1, u, hn = problem("fp32", 80, 2, 700)
    v = u.copy()
    v[1, 400] = bad
    with parament.Parament("fp32") as ctx:
        ctx.set_hamiltonian(H0, *H1)
        ok = ctx.equiprop(0.9 / hn, *u)
        assert np.isnan(ctx.equiprop(0.9 / hn, *v)).all()
        assert np.array_equal(ctx.equiprop(0.9 / hn, *u), ok)
