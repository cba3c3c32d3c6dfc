"""Exact sliced products (fx.cu): complex128, d >= 17 (and complex64, d > 64, below), against the oracle's
FP64 arithmetic: tile edges (17, 63, 64, 65, 128, 129), chunk counts around the
number of SMs and the batch length, every evaluation of the polynomial (powers
in X^2 and X^3, Clenshaw above x = 1, manual orders), non-Hermitian matrices and
complex controls, the device entry point, and samples that are not finite.

Tolerance: both sides round each step's propagator to a few units of 2^-53, the
oracle's J_0(x) the same way at every step: 4e-16 per step, and 4e-15 for the
products of the chunks.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def tol(P):
    return 4e-16 * P + 4e-15


def relerr(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def problem(d, K, n, norm0, hermitian=True, seed=0):
    rng = np.random.default_rng((d, n, seed))

    def h(norm):
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        if hermitian:
            a = a + a.conj().T
        return a * norm / (4 * np.sqrt(d))

    return h(norm0), np.stack([h(1.0) for _ in range(K)]), rng.standard_normal((K, n))


def propagate(H0, H1, u, dt, magnus=False, quad="none", cycles=None):
    import parament_gb300 as parament
    with parament.Parament("fp64") as ctx:
        ctx.set_hamiltonian(H0, *H1, use_magnus=magnus, quadrature_mode=quad)
        if cycles:
            ctx.set_iteration_cycles_manually(cycles)
        U = ctx.equiprop(dt, *u)
        return U, ctx.last_iteration_cycles


@pytest.mark.parametrize("d", [17, 63, 64, 65, 128, 129])
@pytest.mark.parametrize("P,quad,magnus", [(1, "none", False), (3, "midpoint", False), (153, "simpson", False),
                                           (305, "simpson", True)])
def test_tile_and_chunk_edges(built_lib, d, P, quad, magnus):
    n = 2 * P + 1 if quad == "simpson" else P + (quad == "midpoint")
    H0, H1, u = problem(d, 3, n, 6.0)
    U, M = propagate(H0, H1, u, 1e-3, magnus, quad)
    mode = {"none": oracle.NONE, "midpoint": oracle.MIDPOINT, "simpson": oracle.SIMPSON}[quad]
    Uo, Mo = oracle.equiprop(H0, H1, u, 1e-3, magnus=magnus, mode=mode)[:2]
    assert M == Mo
    assert relerr(U, Uo) < tol(P)


@pytest.mark.parametrize("d", [48, 72])
@pytest.mark.parametrize("dt,cycles", [(1e-6, None), (2e-4, None), (2e-3, None), (8e-3, None), (2e-2, None),
                                       (5e-2, None), (0.25, None), (1e-3, 3), (1e-3, 5), (1e-3, 9), (1e-3, 11),
                                       (1e-3, 13), (1e-3, 15), (1e-3, 63), (0.1, 21)])
def test_orders(built_lib, d, dt, cycles):
    H0, H1, u = problem(d, 2, 5, 3.0)
    U, M = propagate(H0, H1, u / 2, dt, cycles=cycles)
    kw = dict(M=cycles) if cycles else {}
    Uo, Mo = oracle.equiprop(H0, H1, u / 2, dt, **kw)[:2]
    assert M == Mo
    assert relerr(U, Uo) < tol(5)


@pytest.mark.parametrize("d,P", [(40, 6000), (80, 40)])
def test_long_and_batched(built_lib, d, P):
    """More steps per chunk than one batch holds (d <= 64: 32; d > 64: 1)."""
    H0, H1, u = problem(d, 2, P, 5.0)
    U, _ = propagate(H0, H1, u, 1e-4)
    assert relerr(U, oracle.equiprop(H0, H1, u, 1e-4)[0]) < tol(P)


@pytest.mark.parametrize("d", [30, 90])
def test_general_matrices_and_complex_controls(built_lib, d):
    H0, H1, u = problem(d, 20, 33, 2.0, hermitian=False)
    u = (u + 1j * np.roll(u, 1, axis=1)) * 10.0 ** (np.arange(20) % 7 - 4)[:, None]
    U, _ = propagate(H0, H1, u / 20, 1e-4)
    assert relerr(U, oracle.equiprop(H0, H1, u / 20, 1e-4)[0]) < tol(33)


def test_graded_and_zero_matrices(built_lib):
    """Levels over eight decades; controls that are zero matrices."""
    d = 36
    H0, H1, u = problem(d, 2, 20, 1e-3)
    H0 = H0 + np.diag(10.0 ** np.linspace(-6, 2, d))
    H1[1] = 0.0
    U, _ = propagate(H0, H1, u, 1e-3)
    assert relerr(U, oracle.equiprop(H0, H1, u, 1e-3)[0]) < tol(20)


@pytest.mark.parametrize("d", [20, 70])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_samples_that_are_not_finite(built_lib, d, bad):
    """One such sample makes the whole propagator NaN, as in FP64 arithmetic,
    and leaves nothing behind for the next call."""
    import parament_gb300 as parament
    H0, H1, u = problem(d, 2, 9, 2.0)
    v = u.copy()
    v[1, 4] = bad
    with parament.Parament("fp64") as ctx:
        ctx.set_hamiltonian(H0, *H1)
        assert np.isnan(ctx.equiprop(1e-3, *v)).all()
        assert relerr(ctx.equiprop(1e-3, *u), oracle.equiprop(H0, H1, u, 1e-3)[0]) < tol(9)


def test_device_entry_point_and_reuse(built_lib):
    """Device tensors on a side stream, a longer and a shorter call on one context."""
    import torch

    import parament_gb300 as parament
    H0, H1, u = problem(64, 2, 700, 4.0)
    with parament.Parament("fp64") as ctx:
        ctx.set_hamiltonian(H0, *H1)
        st = torch.cuda.Stream()
        for P in (700, 1, 31):
            x = torch.tensor(u[:, :P] + 0j, device="cuda")
            torch.cuda.synchronize()
            U = ctx.equiprop_device(1e-3, x, stream=st)
            ctx.synchronize()
            assert relerr(U.cpu().numpy(), oracle.equiprop(H0, H1, u[:, :P], 1e-3)[0]) < tol(P)


# ------------------------------------------------------------------ complex64, d > 64

def c64(*arrays):
    return [np.asarray(a).astype(np.complex64).astype(np.complex128) for a in arrays]


def propagate32(H0, H1, u, dt, magnus=False, quad="none", cycles=None, form="plain"):
    import parament_gb300 as parament
    with parament.Parament("fp32") as ctx:
        ctx.set_precision_mode(form)
        ctx.set_hamiltonian(H0, *H1, use_magnus=magnus, quadrature_mode=quad)
        if cycles:
            ctx.set_iteration_cycles_manually(cycles)
        U = ctx.equiprop(dt, *u)
        return U.astype(np.complex128), ctx.last_iteration_cycles


@pytest.mark.parametrize("d", [65, 96, 128, 129, 200, 300])
@pytest.mark.parametrize("P,quad,magnus", [(1, "none", False), (2, "midpoint", False), (21, "simpson", True)])
@pytest.mark.parametrize("form", ["plain", "split"])
def test_complex64_forms_above_64(built_lib, d, P, quad, magnus, form):
    """The plain form within 1e-5 of the oracle at the complex64 order, the split
    form within 1e-6 of the FP64 oracle at its order (the bars of these forms)."""
    n = 2 * P + 1 if quad == "simpson" else P + (quad == "midpoint")
    H0, H1, u = c64(*problem(d, 2, n, 4.0))
    U, M = propagate32(H0, H1, u, 1e-3, magnus, quad, form=form)
    mode = {"none": oracle.NONE, "midpoint": oracle.MIDPOINT, "simpson": oracle.SIMPSON}[quad]
    Uo, Mo = oracle.equiprop(H0, H1, u, 1e-3, magnus=magnus, mode=mode, single=form == "plain",
                             M=M if form == "split" else 0)[:2]
    assert M == Mo
    assert relerr(U, Uo) < (1e-5 if form == "plain" else 1e-6)


@pytest.mark.parametrize("dt,cycles", [(1e-5, None), (1e-3, None), (1e-2, None), (4e-2, None), (0.1, None),
                                       (1e-3, 3), (1e-3, 7), (1e-3, 9), (1e-3, 15)])
def test_complex64_orders_above_64(built_lib, dt, cycles):
    """Powers of X up to x = 1, the Clenshaw kernels above."""
    H0, H1, u = c64(*problem(80, 2, 5, 3.0))
    U, M = propagate32(H0, H1, u / 2, dt, cycles=cycles)
    Uo, Mo = oracle.equiprop(H0, H1, u / 2, dt, single=True, M=cycles or 0)[:2]
    assert M == Mo
    assert relerr(U, Uo) < 1e-5


@pytest.mark.parametrize("form", ["plain", "split"])
def test_complex64_general_matrices_and_complex_controls(built_lib, form):
    H0, H1, u = problem(90, 18, 17, 2.0, hermitian=False)
    H0, H1, u = c64(H0, H1, (u + 1j * np.roll(u, 1, axis=1)) / 20)
    U, M = propagate32(H0, H1, u, 1e-4, form=form)
    Uo = oracle.equiprop(H0, H1, u, 1e-4, single=form == "plain", M=M)[0]
    assert relerr(U, Uo) < (1e-5 if form == "plain" else 1e-6)


@pytest.mark.parametrize("form", ["plain", "split"])
def test_complex64_samples_that_are_not_finite(built_lib, form):
    H0, H1, u = c64(*problem(70, 2, 9, 2.0))
    u[1, 4] = np.nan
    assert np.isnan(propagate32(H0, H1, u, 1e-3, form=form)[0]).all()
