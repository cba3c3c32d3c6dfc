"""The reduction of an ensemble's chunk products in segments, at the numbers of
chunks where the segments change: one chunk, a short last segment of one, exact
squares, one more than a square.

A lone problem of fewer steps than the device has resident CTAs gets one chunk
per step.  complex128 agrees with the oracle to 1e-10, complex64 with the
single-problem path to 1e-5, as the other ensemble tests.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 3, 4, 5, 9, 10, 16, 17, 151]


@pytest.mark.parametrize("d", [4, 16, 17, 33, 64])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp32", 1e-5)])
def test_ensemble_segments(built_lib, precision, tol, d):
    import parament_gb300 as parament
    from parament_gb300.ensemble import Ensemble
    from parament_gb300.workloads import hermitian, sinusoid_controls
    rng = np.random.default_rng(d)
    for pts in COUNTS:
        H0 = hermitian(rng, d, 1.5)
        H1 = np.stack([hermitian(rng, d, 1.0) for _ in range(2)])
        c = sinusoid_controls(rng, 2, pts, 1e-2)
        with Ensemble([(H0, H1, 1e-2, pts)], precision, "none") as ens:
            ens.set_samples([c])
            U = np.asarray(ens.run()[0])
        if precision == "fp64":
            ref = oracle.equiprop(H0, H1, c, 1e-2, mode=oracle.NONE)[0]
        else:
            with parament.Parament("fp32") as ctx:
                ctx.set_hamiltonian(H0, *H1)
                ref = ctx.equiprop(1e-2, *c)
        assert np.linalg.norm(U - ref) / np.linalg.norm(ref) < tol, pts
