"""Where a few steps of a low order stay with the FP32 and FP64 kernels (fx_faster in
fx.cu): there a context gives, bit for bit, what it gives with the tensor cores
switched off in a child process; beyond the line the sliced products run, which
differ in the last bits.  Both sides stay within the bars of their contexts.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# precision, form, d, steps, x = Hnorm h, below the line
CASES = [
    ("fp32", "plain", 65, 2048, 0.03, True), ("fp32", "plain", 96, 700, 0.03, True),
    ("fp32", "plain", 96, 700, 0.6, False), ("fp32", "plain", 128, 64, 0.2, True), ("fp32", "plain", 128, 200, 0.2, False),
    ("fp32", "plain", 200, 8, 0.2, True), ("fp32", "plain", 200, 40, 0.2, False), ("fp32", "plain", 500, 1, 0.03, True),
    ("fp32", "plain", 500, 3, 0.2, False), ("fp32", "split", 65, 18, 0.2, True), ("fp32", "split", 65, 19, 0.2, False),
    ("fp32", "split", 129, 4, 0.2, True), ("fp32", "split", 129, 5, 0.2, False), ("fp32", "split", 300, 1, 0.2, True),
    ("fp32", "split", 300, 2, 0.2, False), ("fp64", "plain", 17, 150, 0.005, True), ("fp64", "plain", 20, 1, 0.04, True),
    ("fp64", "plain", 20, 400, 0.005, False), ("fp64", "plain", 21, 9, 0.005, False), ("fp64", "plain", 32, 5, 1e-4, True),
    ("fp64", "plain", 33, 5, 1e-4, False), ("fp64", "plain", 18, 9, 0.6, False)]


def problem(precision, d, steps, x):
    rng = np.random.default_rng((d, steps))
    ct = np.complex64 if precision == "fp32" else np.complex128

    def h():
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        return ((a + a.conj().T) / (4 * np.sqrt(d))).astype(ct)

    H0, H1 = h(), np.stack([h() for _ in range(2)])
    u = rng.uniform(-1.0, 1.0, (2, steps)).astype(ct)
    return H0, H1, u, x / float(sum(np.abs(m).sum(0).max() for m in (H0, *H1)))


def solve(precision, form, d, steps, x):
    import parament_gb300 as parament
    H0, H1, u, dt = problem(precision, d, steps, x)
    with parament.Parament(precision) as ctx:
        if form == "split":
            ctx.set_precision_mode("split")
        ctx.set_hamiltonian(H0, *H1)
        return ctx.equiprop(dt, *u), ctx.last_iteration_cycles


@pytest.fixture(scope="module")
def switched_off(built_lib, tmp_path_factory):
    """The results of all cases with the tensor cores switched off."""
    out = str(tmp_path_factory.mktemp("routes") / "off.npz")
    code = ("import sys; sys.path[:0] = [%r, %r]\n" % (ROOT, os.path.join(ROOT, "tests")) +
            "import numpy as np, test_gpu_routes as t\n"
            "np.savez(sys.argv[1], *[t.solve(*c[:5])[0] for c in t.CASES])\n")
    r = subprocess.run([sys.executable, "-c", code, out], cwd=ROOT, capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, PARAMENT_DISABLE_TENSOR_CORES="1"))
    assert r.returncode == 0, r.stderr
    z = np.load(out)
    return [z[f"arr_{i}"] for i in range(len(CASES))]


@pytest.mark.parametrize("i", range(len(CASES)))
def test_line(switched_off, i):
    precision, form, d, steps, x, below = CASES[i]
    U, M = solve(precision, form, d, steps, x)
    assert np.array_equal(U, switched_off[i]) == below
    if d * d * d * steps <= 2e8:
        H0, H1, u, dt = problem(precision, d, steps, x)
        c = [a.astype(np.complex128) for a in (H0, H1, u)]
        Uo, Mo = oracle.equiprop(*c, dt, single=precision == "fp32" and form == "plain", M=M if form == "split" else 0)[:2]
        assert M == Mo
        bar = {"plain": 1e-5 if precision == "fp32" else 1e-10, "split": 1e-6}[form]
        assert np.linalg.norm(U - Uo) / np.linalg.norm(Uo) < bar


@pytest.mark.parametrize("precision,d,steps,launches", [
    ("fp64", 8, 1, 0), ("fp64", 5, 8, 0), ("fp64", 8, 9, 1), ("fp64", 4, 2, 1), ("fp32", 8, 2, 1)])
@pytest.mark.parametrize("x", [1e-4, 0.6])
def test_small_groups(built_lib, precision, d, steps, launches, x):
    """d <= 8: one launch in all, or (complex128, d > 4, up to eight steps) the step
    kernel and the tree, as many as a call above x = 1 takes."""
    import parament_gb300 as parament
    H0, H1, u, dt = problem(precision, d, steps, x)
    with parament.Parament(precision) as ctx:
        ctx.set_hamiltonian(H0, *H1)
        count = ctx._fn("Parament_lastLaunchCount")
        ctx.equiprop(dt / x * 1.5, *u)
        above = int(count(ctx._handle))
        U = ctx.equiprop(dt, *u)
        assert int(count(ctx._handle)) == (launches or above)
    c = [a.astype(np.complex128) for a in (H0, H1, u)]
    Uo = oracle.equiprop(*c, dt, single=precision == "fp32")[0]
    assert np.linalg.norm(U - Uo) / np.linalg.norm(Uo) < (1e-5 if precision == "fp32" else 1e-14)
