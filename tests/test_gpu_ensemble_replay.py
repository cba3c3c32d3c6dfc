"""Replays of an ensemble's graph give the same bits: problems of all dimension
classes, the first run against the later ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("seed", [2, 4, 6, 9])
def test_replays_agree(built_lib, precision, seed):
    from parament_gb300.ensemble import Ensemble
    from parament_gb300.workloads import hermitian, sinusoid_controls
    rng = np.random.default_rng(seed)
    dims = [2, 3, 4, 5, 7, 8, 12, 16, 20, 31, 32, 40, 63, 64]
    probs = []
    for i in range(40):
        d, K, pts = dims[i % len(dims)], int(rng.integers(1, 5)), int(rng.integers(3, 400))
        H0 = hermitian(rng, d, float(rng.uniform(0.5, 3.0)))
        H1 = np.stack([hermitian(rng, d, 1.0) for _ in range(K)])
        probs.append((H0, H1, 1e-2, sinusoid_controls(rng, K, pts, 1e-2)))
    with Ensemble([(H0, H1, dt, c.shape[1]) for H0, H1, dt, c in probs], precision, "none") as ens:
        ens.set_samples([c for *_, c in probs])
        first = [np.array(U) for U in ens.run()]
        for _ in range(20):
            for i, (a, b) in enumerate(zip(first, ens.run())):
                assert np.array_equal(a, b), (probs[i][0].shape[0], len(probs[i][1]), probs[i][3].shape[1])
