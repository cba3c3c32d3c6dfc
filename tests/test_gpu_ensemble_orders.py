"""Ensembles at the orders and norms where the polynomial of a step changes its
form: order 3 (recurrence), the first orders by powers of X, a norm just below and
just above 1 (recurrence again), in each dimension class.

complex128 agrees with the oracle to 1e-10, complex64 with the single-problem path
to 1e-5, as the other ensemble tests.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NORMS = [0.01, 0.1, 0.3, 0.6, 0.99, 1.01, 2.0]


@pytest.mark.parametrize("d", [1, 4, 5, 8, 13, 16, 27, 32, 50, 64])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp32", 1e-5)])
def test_ensemble_orders(built_lib, precision, tol, d):
    import parament_gb300 as parament
    from parament_gb300.ensemble import Ensemble
    from parament_gb300.workloads import hermitian
    rng = np.random.default_rng(100 + d)
    pts = 24
    probs = []
    for x in NORMS:
        H0 = hermitian(rng, d, 1.0)
        H1 = np.stack([hermitian(rng, d, 1.0) for _ in range(2)])
        hn = sum(np.abs(m).sum(0).max() for m in (H0, *H1))
        probs.append((H0, H1, x / hn, rng.uniform(-1.0, 1.0, (2, pts))))
    with Ensemble([(H0, H1, dt, pts) for H0, H1, dt, _ in probs], precision, "none") as ens:
        ens.set_samples([c for *_, c in probs])
        Us = [np.asarray(U) for U in ens.run()]
    for x, (H0, H1, dt, c), U in zip(NORMS, probs, Us):
        if precision == "fp64":
            ref = oracle.equiprop(H0, H1, c, dt, mode=oracle.NONE)[0]
        else:
            with parament.Parament("fp32") as ctx:
                ctx.set_hamiltonian(H0, *H1)
                ref = ctx.equiprop(dt, *c)
        assert np.linalg.norm(U - ref) / np.linalg.norm(ref) < tol, x
