"""complex128 with manual orders at steps far beyond what the order resolves: the same
polynomial as the oracle's, whose coefficient J_0(x) the fixed-point kernels take as
J_0 - 1.  Off by a few units of 2^-53 of the identity's norm per product of the
recurrence.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [36, 72])
@pytest.mark.parametrize("x", [1.5, 2.5, 7.9, 8.1, 30.0, 55.0, 1000.0])
@pytest.mark.parametrize("cycles", [3, 9, 13])
def test_manual_orders(built_lib, d, x, cycles):
    import parament_gb300 as parament
    rng = np.random.default_rng((d, cycles))

    def h():
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        return (a + a.conj().T) / (4 * np.sqrt(d))

    H0, H1, u = h(), h()[None], rng.uniform(-1.0, 1.0, (1, 1))
    hn = sum(np.abs(m).sum(0).max() for m in (H0, *H1))
    with parament.Parament("fp64") as ctx:
        ctx.set_hamiltonian(H0, *H1)
        ctx.set_iteration_cycles_manually(cycles)
        U = ctx.equiprop(x / hn, *u)
    Uo = oracle.equiprop(H0, H1, u, x / hn, M=cycles)[0]
    assert np.linalg.norm(U - Uo) / np.sqrt(d) < 2e-16 * (cycles + 10)
