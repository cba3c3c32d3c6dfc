"""Propagations of small problems: groups of threads (step_group.cu, d <= 8) and the
kernels that follow above, against the oracle: dimensions at the edges of the
micro-tiles (odd ones too), chunk counts with and without a partner on every level
of the tree that runs inside the launch (d <= 8), the orders, general matrices and
complex controls, stacks too large for shared memory, calls of different length on
one context (the pair counters return to zero) and the hand-over to the FP64 /
Clenshaw kernels above x = 1.

Tolerances: complex128 4e-16 per step and 4e-15 for the rest (both sides round a
step's propagator to a few units of 2^-53); complex64 1e-5, the bar of the
complex64 contexts, over at most 1217 steps.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def tol(precision, P):
    return 1e-5 if precision == "fp32" else 4e-16 * P + 4e-15


def relerr(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def problem(precision, d, K, n, norm0, hermitian=True):
    rng = np.random.default_rng((d, n, K))

    def h(norm):
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        if hermitian:
            a = a + a.conj().T
        return a * norm / (4 * np.sqrt(d))

    H0, H1, u = h(norm0), np.stack([h(1.0) for _ in range(K)]), rng.standard_normal((K, n)) + 0j
    if precision == "fp32":
        H0, H1, u = (x.astype(np.complex64).astype(np.complex128) for x in (H0, H1, u))
    return H0, H1, u


def reference(precision, H0, H1, u, dt, magnus=False, quad="none", cycles=0):
    mode = {"none": oracle.NONE, "midpoint": oracle.MIDPOINT, "simpson": oracle.SIMPSON}[quad]
    return oracle.equiprop(H0, H1, u, dt, magnus=magnus, mode=mode, single=precision == "fp32", M=cycles)[:2]


def propagate(precision, H0, H1, u, dt, magnus=False, quad="none", cycles=0):
    import parament_gb300 as parament
    with parament.Parament(precision) as ctx:
        ctx.set_hamiltonian(H0, *H1, use_magnus=magnus, quadrature_mode=quad)
        if cycles:
            ctx.set_iteration_cycles_manually(cycles)
        U = ctx.equiprop(dt, *u)
        return U.astype(np.complex128), ctx.last_iteration_cycles


DIMS = [("fp32", d) for d in (1, 2, 3, 4, 5, 7, 8, 9, 16, 17, 31, 32)] + \
       [("fp64", d) for d in (1, 2, 3, 4, 5, 8, 9, 15, 16)]


@pytest.mark.parametrize("precision,d", DIMS)
@pytest.mark.parametrize("P,quad,magnus", [(1, "none", False), (2, "midpoint", False), (7, "simpson", True),
                                           (100, "simpson", False), (1217, "none", False)])
def test_dimensions_and_chunk_counts(built_lib, precision, d, P, quad, magnus):
    n = 2 * P + 1 if quad == "simpson" else P + (quad == "midpoint")
    H0, H1, u = problem(precision, d, 2, n, 3.0)
    U, M = propagate(precision, H0, H1, u, 1e-3, magnus, quad)
    Uo, Mo = reference(precision, H0, H1, u, 1e-3, magnus, quad)
    assert M == Mo
    assert relerr(U, Uo) < tol(precision, P)


@pytest.mark.parametrize("precision,d", [("fp32", 3), ("fp32", 13), ("fp32", 27), ("fp64", 6), ("fp64", 14)])
@pytest.mark.parametrize("dt,cycles", [(1e-5, 0), (5e-3, 0), (3e-2, 0), (0.1, 0), (0.6, 0), (1e-3, 3), (1e-3, 9),
                                       (1e-3, 63), (1e-3, 1)])
def test_orders(built_lib, precision, d, dt, cycles):
    H0, H1, u = problem(precision, d, 1, 9, 1.5)
    U, M = propagate(precision, H0, H1, u / 3, dt, cycles=cycles)
    Uo, Mo = reference(precision, H0, H1, u / 3, dt, cycles=cycles)
    assert M == Mo
    assert relerr(U, Uo) < tol(precision, 9)


@pytest.mark.parametrize("precision,d,K,magnus", [("fp32", 6, 20, True), ("fp32", 32, 12, True), ("fp32", 21, 40, False),
                                                  ("fp64", 8, 70, False), ("fp64", 16, 9, True)])
def test_many_controls_general_matrices(built_lib, precision, d, K, magnus):
    """Non-Hermitian matrices, complex controls, stacks in and out of shared memory."""
    H0, H1, u = problem(precision, d, K, 43, 2.0, hermitian=False)
    u = (u + 1j * np.roll(u, 1, axis=1)) / 16
    quad = "simpson" if magnus else "none"
    U, _ = propagate(precision, H0, H1, u, 2e-4, magnus, quad)
    assert relerr(U, reference(precision, H0, H1, u, 2e-4, magnus, quad)[0]) < tol(precision, 43)


@pytest.mark.parametrize("precision,d", [("fp32", 2), ("fp32", 8), ("fp32", 20), ("fp64", 4), ("fp64", 12)])
def test_calls_of_different_length_on_one_context(built_lib, precision, d):
    """A call leaves nothing behind: bit for bit the result of a context of its own."""
    import parament_gb300 as parament
    H0, H1, u = problem(precision, d, 2, 3000, 2.0)

    def context():
        ctx = parament.Parament(precision)
        ctx.set_hamiltonian(H0, *H1)
        return ctx

    with context() as ctx:
        for P in (40, 3000, 1, 40, 777):
            U = ctx.equiprop(1e-4, *u[:, :P])
            with context() as fresh:
                assert np.array_equal(U, fresh.equiprop(1e-4, *u[:, :P]))
