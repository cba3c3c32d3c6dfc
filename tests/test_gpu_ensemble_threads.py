"""Ensembles of several host threads at once, each on its own stream: one of d = 16 alone
and two of d <= 8, whose kernels then share the SMs.  Every run of each gives, bit for
bit, what the ensemble gives alone.
"""
import numpy as np
import pytest

from test_gpu_threads import problem, together

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,repeats", [("fp32", 1500), ("fp64", 250)])
def test_runs_beside_each_other(built_lib, precision, repeats):
    from parament_gb300.ensemble import Ensemble

    def job(dims, seed):
        rng = np.random.default_rng(seed)
        probs = [problem(precision, int(d), int(rng.integers(1, 5)), int(rng.integers(3, 4000)))
                 for d in rng.choice(dims, 60)]
        ens = Ensemble([(H0, H1, 1e-2, u.shape[1]) for H0, H1, u in probs], precision, "none")
        ens.set_samples([u for *_, u in probs])
        ref = [np.array(U) for U in ens.run()]

        def run():
            for _ in range(repeats):
                for (H0, _, u), a, b in zip(probs, ref, ens.run()):
                    assert np.array_equal(a, b), (H0.shape[0], u.shape, np.argwhere(a != b)[:4].tolist())

        return run

    together(job([16], 1), job([2, 3, 4, 5, 7, 8], 2), job([5, 8], 3))
