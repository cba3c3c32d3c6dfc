"""Hamiltonians in other units than those of order one (rad/s, joules): times a
power of two, with the step length divided by it, a propagator and its gradient are
the same bits, whatever the order, dimension and form; and at decimal norms the
complex64 and complex128 results keep the bars of their contexts (1e-5 and 1e-10 of
the oracle).

The powers of two are exact in every product, sum and coefficient as long as nothing
leaves the range of the type, so the comparison has no tolerance.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# x = Hnorm h for orders 3, 5, 7, 9 of the complex64 table (complex128: 7 .. 15), and one
# above 1, where the recurrence runs.
XS = [0.02, 0.15, 0.5, 0.95, 1.5]
POWERS = {"fp32": [-27, 20, 33, 50], "fp64": [-80, -27, 50, 200]}


def problem(precision, d, K, pts, magnus=False):
    rng = np.random.default_rng((d, K, pts))
    ct = np.complex64 if precision == "fp32" else np.complex128

    def h():
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        return ((a + a.conj().T) / (4 * np.sqrt(d))).astype(ct)

    n = 2 * pts + 1 if magnus else pts
    u = rng.uniform(-1.0, 1.0, (K, n)).astype(ct)
    W = (rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))).astype(ct)
    return h(), np.stack([h() for _ in range(K)]), u, W


def times(a, q):
    """a 2^q, exactly."""
    out = np.empty_like(a)
    out.real, out.imag = np.ldexp(a.real, q), np.ldexp(a.imag, q)
    return out


def run(precision, H0, H1, u, dt, W=None, magnus=False, form="plain"):
    import parament_gb300 as parament
    with parament.Parament(precision) as ctx:
        if form == "split":
            ctx.set_precision_mode("split")
        ctx.set_hamiltonian(H0, *H1, use_magnus=magnus, quadrature_mode="simpson" if magnus else "none")
        U = ctx.equiprop(dt, *u)
        g = ctx.vjp(dt, W, *u) if W is not None else None
        return U, g, ctx.last_iteration_cycles, ctx.hamiltonian_norm


def step(H0, H1, x, magnus):
    """The sample distance with Hnorm h = x (a Magnus step spans two)."""
    hn = sum(np.abs(m.astype(np.complex128)).sum(0).max() for m in (H0, *H1))
    return x / hn / (2 if magnus else 1)


@pytest.mark.parametrize("precision,d", [("fp32", d) for d in (2, 8, 12, 16, 32, 64, 72, 256)] +
                         [("fp64", d) for d in (2, 8, 16, 32, 64, 72)])
@pytest.mark.parametrize("magnus", [False, True])
def test_powers_of_two_change_no_bit(built_lib, precision, d, magnus):
    H0, H1, u, W = problem(precision, d, 2, 5, magnus)
    grad = d <= (64 if precision == "fp32" else 48)
    for x in XS:
        dt = step(H0, H1, x, magnus)
        U, g, M, hn = run(precision, H0, H1, u, dt, W if grad else None, magnus)
        assert np.isfinite(U).all()
        for q in POWERS[precision]:
            V, k, N, hq = run(precision, times(H0, q), times(H1, q), u, float(np.ldexp(dt, -q)), W if grad else None,
                              magnus)
            assert N == M and hq == np.ldexp(hn, q)
            assert np.array_equal(U, V), (x, q)
            if grad:
                assert np.isfinite(g).all() and np.array_equal(g, k), (x, q)


@pytest.mark.parametrize("d", [3, 20, 64, 72])
@pytest.mark.parametrize("magnus", [False, True])
def test_split_form(built_lib, d, magnus):
    H0, H1, u, _ = problem("fp32", d, 2, 5, magnus)
    for x in (0.02, 0.15, 0.45):
        dt = step(H0, H1, x, magnus)
        U = run("fp32", H0, H1, u, dt, None, magnus, "split")[0]
        for q in POWERS["fp32"]:
            V = run("fp32", times(H0, q), times(H1, q), u, float(np.ldexp(dt, -q)), None, magnus, "split")[0]
            assert np.array_equal(U, V), (x, q)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_ensembles(built_lib, precision):
    from parament_gb300.ensemble import Ensemble
    probs = [(problem(precision, d, 2, 9), x) for d in (2, 7, 16, 30, 64) for x in XS]

    def solve(q):
        sc = [(times(H0, q), times(H1, q), float(np.ldexp(step(H0, H1, x, False), -q)), u.shape[1])
              for (H0, H1, u, _), x in probs]
        with Ensemble(sc, precision, "none") as ens:
            ens.set_samples([u for (_, _, u, _), _ in probs])
            return [np.array(U) for U in ens.run()]

    ref = solve(0)
    for q in POWERS[precision]:
        for (p, x), U, V in zip(probs, ref, solve(q)):
            assert np.isfinite(U).all() and np.array_equal(U, V), (p[0].shape[0], x, q)


@pytest.mark.parametrize("d", [2, 8, 16, 64])
@pytest.mark.parametrize("precision,bar", [("fp32", 1e-5), ("fp64", 1e-10)])
def test_decimal_norms_against_the_oracle(built_lib, precision, bar, d):
    """Twelve steps, each off by at most a few units of 2^-24 (1 + x): 5e-6."""
    H0, H1, u, _ = problem(precision, d, 2, 12)
    for norm in (1e-8, 1e6, 1e10, 1e15):
        H0s, H1s = (H0 * norm).astype(H0.dtype), (H1 * norm).astype(H0.dtype)
        for x in XS:
            dt = step(H0s, H1s, x, False)
            U, _, M, _ = run(precision, H0s, H1s, u, dt)
            Uo, Mo = oracle.equiprop(H0s.astype(np.complex128), H1s.astype(np.complex128), u.astype(np.complex128), dt,
                                     single=precision == "fp32")[:2]
            assert M == Mo
            assert np.linalg.norm(U - Uo) / np.linalg.norm(Uo) < bar, (norm, x)


def test_no_alloc_entry_point(built_lib):
    import ctypes

    import torch

    lib = ctypes.CDLL(built_lib)
    vp = ctypes.c_void_p
    lib.Parament_equipropNoAlloc_fp64.argtypes = [vp, vp, ctypes.c_double, ctypes.c_uint, ctypes.c_uint, vp, vp]
    import parament_gb300 as parament
    for d in (5, 20):
        H0, H1, u, _ = problem("fp64", d, 2, 30)
        ref = None
        for q in (0, -80, 200):
            dt = float(np.ldexp(step(H0, H1, 0.95, False), -q))
            with parament.Parament("fp64") as ctx:
                ctx.set_hamiltonian(times(H0, q), *times(H1, q))
                carr = torch.from_numpy(u).cuda()
                out = torch.empty((d, d), dtype=torch.complex128, device="cuda")
                torch.cuda.synchronize()
                assert lib.Parament_equipropNoAlloc_fp64(ctx._handle, carr.data_ptr(), dt, 30, 2, out.data_ptr(),
                                                         None) == 0
                torch.cuda.synchronize()
                U = out.cpu().numpy()
            ref = U if ref is None else ref
            assert np.isfinite(U).all() and np.array_equal(U, ref)
