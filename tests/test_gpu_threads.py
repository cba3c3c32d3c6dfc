"""Contexts of several host threads at once, each thread with its own
(as the library asks): no call fails and every result is, bit for bit, the one the
same object gives alone.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def together(*jobs):
    """Runs the jobs, each in a thread, and raises what any of them raised."""
    errors = []

    def guarded(job):
        try:
            job()
        except BaseException as e:  # noqa: B036
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def problem(precision, d, K, pts):
    rng = np.random.default_rng((d, K, pts))
    ct = np.complex64 if precision == "fp32" else np.complex128

    def h():
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        return ((a + a.conj().T) / (4 * np.sqrt(d))).astype(ct)

    return h(), [h() for _ in range(K)], rng.uniform(-1.0, 1.0, (K, pts)).astype(ct)


@pytest.mark.parametrize("precision,small,large", [
    # One kernel, two sizes of its dynamic shared memory (by d, controls and steps).
    ("fp32", (6, 1, 3), (8, 40, 4000)), ("fp64", (5, 1, 3), (8, 30, 4000)), ("fp32", (33, 1, 40), (48, 6, 40)),
    ("fp64", (9, 1, 40), (16, 30, 40))])
@pytest.mark.parametrize("grad", [False, True])
def test_contexts(built_lib, precision, small, large, grad):
    import parament_gb300 as parament

    def job(size, dt=1e-3):
        H0, H1, u = problem(precision, *size)
        W = np.eye(size[0], dtype=u.dtype)
        ctx = parament.Parament(precision)
        ctx.set_hamiltonian(H0, *H1)

        def call():
            return ctx.vjp(dt, W, *u) if grad else ctx.equiprop(dt, *u)

        ref = call()

        def run():
            for _ in range(150):
                assert np.array_equal(call(), ref)

        return run

    together(job(small), job(large))
