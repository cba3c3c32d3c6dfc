"""The backward sweep by powers of X (k_adj_sweep: automatic order, x = Hnorm h <= 1)
against the stored-checkpoint kernel (manual order, set to the same value), which
shares none of its products: every order up to x = 1 and the hand-over above,
dimensions at the edges of the 16-wide tiles, quadratures, and complex64 against
complex128.

Tolerances, relative to the largest entry: complex128 1e-11 (both sum at most 300
steps of FP64 products of factors of norm one); complex64 2e-4 (the bar of the
complex64 gradient tests).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problem(d, K, n, norm0, seed=0):
    rng = np.random.default_rng((d, n, seed))

    def h(norm):
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        return (a + a.conj().T) * norm / (4 * np.sqrt(d))

    W = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
    return h(norm0), np.stack([h(1.0) for _ in range(K)]), rng.standard_normal((K, n)) / 2, W


def gradients(precision, H0, H1, u, W, dt, magnus=False, quad="none"):
    """By the automatic order, and by the same order set by hand."""
    import parament_gb300 as parament
    with parament.Parament(precision) as ctx:
        ctx.set_hamiltonian(H0, *H1, use_magnus=magnus, quadrature_mode=quad)
        g = ctx.vjp(dt, W, *u)
        M = ctx.last_iteration_cycles
        ctx.set_iteration_cycles_manually(M)
        return g.astype(np.float64), ctx.vjp(dt, W, *u).astype(np.float64), M


def off(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("d", [1, 2, 15, 16, 17, 32, 33, 48])
@pytest.mark.parametrize("P,quad,magnus", [(1, "none", False), (9, "midpoint", False), (300, "simpson", True)])
def test_dimensions(built_lib, d, P, quad, magnus):
    n = 2 * P + 1 if quad == "simpson" else P + (quad == "midpoint")
    H0, H1, u, W = problem(d, 3, n, 3.0)
    g, ref, _ = gradients("fp64", H0, H1, u, W, 1e-3, magnus, quad)
    assert off(g, ref) < 1e-11


@pytest.mark.parametrize("dt,order", [(2e-6, 3), (2e-4, 5), (2e-3, 7), (8e-3, 9), (1.6e-2, 11), (3e-2, 13), (6e-2, 15),
                                      (0.15, 21)])
def test_orders(built_lib, dt, order):
    H0, H1, u, W = problem(24, 2, 7, 4.0)
    g, ref, M = gradients("fp64", H0, H1, u, W, dt)
    assert abs(M - order) <= 4
    assert off(g, ref) < 1e-11


@pytest.mark.parametrize("d", [3, 16, 31, 32, 48, 64])
@pytest.mark.parametrize("dt", [1e-4, 2e-3, 1e-2, 4e-2])
def test_complex64(built_lib, d, dt):
    H0, H1, u, W = problem(d, 3, 200, 2.0)
    H0, H1, W = (x.astype(np.complex64).astype(np.complex128) for x in (H0, H1, W))
    u = u.astype(np.float32).astype(np.float64)
    g = gradients("fp32", H0, H1, u, W, dt)[0]
    if d <= 48:
        assert off(g, gradients("fp64", H0, H1, u, W, dt)[0]) < 2e-4
    else:
        assert off(g, gradients("fp32", H0, H1, u, W, dt)[1]) < 2e-4
