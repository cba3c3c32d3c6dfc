"""complex64 steps by powers of X: rounding the regrouped coefficients c_n to FP32 would
turn every step by the same angle.

Diagonal Hamiltonians (each level a product of scalars) whose samples vary, so that what
the arithmetic rounds differs from step to step and adds up like a random walk, while
coefficients round alike at every step.  The reference is the polynomial with FP32 Bessel
functions, as the recurrence has them, in double.  Bar, in units of 2^-24: 4 sqrt(P) for
the arithmetic and P x^3 / 5 for the coefficients from c_3 on.  Rounded c_1 and c_2 give up
to P x / 2 beside it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
P = 16384


@pytest.mark.parametrize("d", [2, 5, 8, 9, 16, 40, 64])
@pytest.mark.parametrize("x", [0.2, 0.26, 0.31, 0.37, 0.4, 0.45])
def test_coefficients_add_no_angle(built_lib, d, x):
    import oracle
    import parament_gb300 as parament
    rng = np.random.default_rng(d)
    h0 = rng.uniform(0.5, 0.8, d).astype(np.float32)
    h1 = rng.uniform(0.05, 0.2, d).astype(np.float32)
    h0[0], h1[0] = 0.8, 0.2
    u = rng.uniform(-1, 1, P).astype(np.float32)
    with parament.Parament("fp32") as ctx:
        ctx.set_hamiltonian(np.diag(h0).astype(np.complex64), np.diag(h1).astype(np.complex64))
        hn = ctx.hamiltonian_norm
        ctx.set_iteration_cycles_manually(7)
        U = ctx.equiprop(x / hn, u.astype(np.complex64))
    J = oracle.bessel_coeffs(7, x).astype(np.complex64).astype(complex)  # (-i)^k J_k
    y = (h0[:, None].astype(float) + u[None, :] * h1[:, None].astype(float)) * (float(np.float32(2.0 / hn)) / 2)
    T = [np.ones_like(y), y]
    v = J[0] + 2 * J[1] * y
    for k in range(2, 8):
        T.append(2 * y * T[-1] - T[-2])
        v = v + 2 * J[k] * T[-1]
    assert np.abs(np.diag(U) - v.prod(1)).max() < 2.0 ** -24 * (4 * np.sqrt(P) + P * x**3 / 5)
