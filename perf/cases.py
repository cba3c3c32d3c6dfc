"""What the framework is measured on: propagators of driven quantum systems,
their gradients and ensembles of them, through the calls a user's program makes.

A case names the entry point (``kind``), the context (``precision``, ``form``),
the problem (``d``, ``K`` controls, ``steps``, ``dt``, the drift's norm
``norm0``; every control Hamiltonian has norm 1) and the quadrature:

* ``host``: ``Parament.equiprop`` on numpy arrays, result in a numpy array;
* ``device``: ``Parament.equiprop_device`` on CUDA tensors;
* ``grad``: ``propagate`` and ``fidelity_loss`` under ``torch.autograd``, one
  pass forward and backward of a gate optimisation;
* ``ensemble``: ``Ensemble.set_samples`` and ``Ensemble.run`` over ``n``
  problems of mixed size.

The context with its Hamiltonians (and the tuned ensemble) is what a program
keeps from call to call; the control samples are what changes.
"""
import math

import numpy as np
import torch

import parament_gb300 as parament
from parament_gb300.autograd import fidelity_loss, propagate
from parament_gb300.ensemble import Ensemble

ENS_DIMS = (4, 8, 16, 32, 64)
ENS_SHARE = (0.3, 0.3, 0.2, 0.15, 0.05)


def _case(name, kind, precision, d, K, steps, norm0=1.0, dt=1e-3, quadrature="none", magnus=False, form="plain"):
    c = dict(kind=kind, precision=precision, form=form, d=d, K=K, steps=steps, norm0=norm0, dt=dt,
             quadrature=quadrature, magnus=magnus)
    return dict(c, name=name) if name else c


def _ensemble(name, n, precision, pts_min, pts_max):
    c = dict(kind="ensemble", n=n, precision=precision, pts_min=pts_min, pts_max=pts_max, dt=1e-3)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One qubit under a short pulse, from a script or a notebook: nothing
        # but the latency of the call.
        _case("qubit_d2", "host", "fp32", 2, 1, 100, dt=0.01),
        # A four-qubit gate in double precision, the plain d = 16 benchmark.
        _case("qubits_d16_fp64", "host", "fp64", 16, 2, 4096),
        # Three qutrits (an odd dimension) with interpolated samples already
        # on the GPU, as an optimiser on the device calls it.
        _case("qutrits_d27", "device", "fp32", 27, 3, 5000, norm0=4.0, quadrature="midpoint"),
        # Six qubits, fourth-order Magnus steps with Simpson's rule: the
        # precision benchmark's problem in each of the three arithmetic forms.
        _case("magnus_d64", "device", "fp32", 64, 4, 8192, norm0=10.0, quadrature="simpson", magnus=True),
        _case("magnus_d64_split", "host", "fp32", 64, 4, 65536, norm0=10.0, quadrature="simpson", magnus=True,
              form="split"),
        _case("magnus_d64_fp64", "host", "fp64", 64, 4, 4096, norm0=10.0, quadrature="simpson", magnus=True),
        # Seven qubits in single precision; a spin-boson-like odd multiple of
        # 32 in double precision with Simpson's rule.
        _case("mid_d128", "device", "fp32", 128, 3, 4096, norm0=8.0),
        _case("mid_d96_fp64", "host", "fp64", 96, 3, 512, norm0=8.0, quadrature="simpson"),
        # Nine qubits with eight smooth controls: the large dense workload.
        _case("dense_d512", "device", "fp32", 512, 8, 64, norm0=20.0),
        _case("dense_d512_fp64", "host", "fp64", 512, 8, 16, norm0=20.0),
        # Gradient of a gate infidelity with respect to every sample: the
        # gradient workload (d = 32, six controls, 16384 steps).
        _case("grape_d32", "grad", "fp32", 32, 6, 16384),
        # Many small problems of uneven size at once, as the ensemble
        # workload: robustness scans over detunings and drive amplitudes.
        _ensemble("ensemble", 512, "fp32", 256, 8192),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("host", "host", "device", "device", "large", "large", "grad", "ensemble"))
    precision = rng.choice(("fp32", "fp32", "fp64"))
    if kind == "ensemble":
        lo = _log_int(rng, 64, 512)
        return _ensemble(None, _log_int(rng, 32, 512 if precision == "fp32" else 64), precision, lo,
                         _log_int(rng, 2 * lo, 16 * lo))
    if kind == "grad":
        d = _log_int(rng, 2, 64 if precision == "fp32" else 48)
        most = 16384 if precision == "fp32" else min(16384, max(64, int(2.5e8 / d ** 3)))
        quadrature, magnus = rng.choice((("none", False), ("midpoint", False), ("simpson", False), ("simpson", True)))
        return _case(None, "grad", precision, d, rng.randint(1, 6), _log_int(rng, 64, most),
                     norm0=round(rng.uniform(1.0, 4.0), 2), quadrature=quadrature, magnus=magnus)
    if kind == "large":
        d = _log_int(rng, 65, 512)
        if rng.random() < 0.4:
            d = 32 * max(3, d // 32)
        form = rng.choice(("plain", "split")) if precision == "fp32" else "plain"
        flops = 1.5e12 if precision == "fp32" else 1.2e11
        most = min(4096 if d <= 128 else 64 if form == "plain" else 512, int(flops / (64.0 * d ** 3)))
        return _case(None, rng.choice(("host", "device")), precision, d, rng.randint(1, 8),
                     _log_int(rng, 8, max(16, most)),
                     # The split form takes steps up to a norm times step length of 0.5.
                     norm0=round(rng.uniform(4.0, 12.0 if form == "split" else 20.0), 2),
                     quadrature=rng.choice(("none", "midpoint", "simpson")), form=form)
    d = _log_int(rng, 2, 64)
    if rng.random() < 0.4:
        d = 1 << max(1, d.bit_length() - 1)
    form = rng.choice(("plain", "plain", "split")) if precision == "fp32" else "plain"
    most = 65536 if form == "split" else 8192 if precision == "fp32" else min(65536, int(1.1e9 / d ** 3))
    quadrature, magnus = rng.choice((("none", False), ("midpoint", False), ("simpson", False), ("simpson", True)))
    return _case(None, kind, precision, d, rng.randint(1, 4), _log_int(rng, 16, most),
                 norm0=round(rng.uniform(1.0, 10.0), 2), quadrature=quadrature, magnus=magnus, form=form)


# ------------------------------------------------------------------ inputs

def _points(case):
    if case["quadrature"] == "simpson":
        return 2 * case["steps"] + 1
    return case["steps"] + (1 if case["quadrature"] == "midpoint" else 0)


def _hermitian(rng, d, norm):
    """A random Hermitian matrix of spectral norm near ``norm`` (the edge of the
    semicircle of its ensemble)."""
    a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
    return (a + a.conj().T) * (norm / (4.0 * math.sqrt(d)))


def _controls(rng, K, n, dt):
    """Sinusoids with a little noise on every sample, as of a pulse generator."""
    f, phi = rng.uniform(1.0, 20.0, (K, 1)), rng.uniform(0.0, 2 * np.pi, (K, 1))
    return np.sin(2 * np.pi * f * (np.arange(n) * dt) + phi) + 0.1 * rng.standard_normal((K, n))


def _problem(case, seed):
    """(H0, H1, samples) as the context's type holds them: complex64 inputs are
    rounded once, here."""
    rng = np.random.default_rng(seed)
    ct = np.complex64 if case["precision"] == "fp32" else np.complex128
    d, K = case["d"], case["K"]
    H0 = _hermitian(rng, d, case["norm0"]).astype(ct)
    H1 = np.stack([_hermitian(rng, d, 1.0) for _ in range(K)]).astype(ct)
    return H0, H1, _controls(rng, K, _points(case), case["dt"]).astype(ct)


def _ensemble_problems(case, seed):
    # The sizes belong to the case; matrices and samples come from the seed.
    sizes, rng = np.random.default_rng((case["n"], case["pts_max"])), np.random.default_rng(seed)
    ct = np.complex64 if case["precision"] == "fp32" else np.complex128
    out = []
    for d in sizes.choice(ENS_DIMS, size=case["n"], p=ENS_SHARE):
        d, K = int(d), int(sizes.integers(1, 5))
        pts = int(sizes.integers(case["pts_min"], case["pts_max"] + 1))
        H0 = _hermitian(rng, d, 1.0) + np.diag(rng.normal(0.0, 0.05, d))
        H1 = np.stack([_hermitian(rng, d, 1.0) for _ in range(K)])
        out.append((H0.astype(ct), H1.astype(ct), _controls(rng, K, pts, case["dt"]).astype(ct)))
    return out


def _unitary(seed, d):
    """The target of the gradient cases: a random unitary."""
    rng = np.random.default_rng(seed + 7919)
    return np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))[0]


def prepare(case, seed):
    if case["kind"] == "ensemble":
        problems = _ensemble_problems(case, seed)
        ens = Ensemble([(H0, H1, case["dt"], u.shape[1]) for H0, H1, u in problems], precision=case["precision"])
        samples = [u for _, _, u in problems]
        ens.set_samples(samples)
        ens.tune()
        return dict(kind="ensemble", ens=ens, samples=samples)
    H0, H1, u = _problem(case, seed)
    ctx = parament.Parament(case["precision"])
    if case["form"] == "split":
        ctx.set_precision_mode("split")
    ctx.set_hamiltonian(H0, *H1, use_magnus=case["magnus"], quadrature_mode=case["quadrature"])
    state = dict(kind=case["kind"], ctx=ctx, dt=case["dt"])
    if case["kind"] == "host":
        state["samples"] = u
    elif case["kind"] == "device":
        state["samples"] = torch.from_numpy(u).cuda()
    else:
        # Real samples of an optimiser; the propagator's type decides theirs.
        state["samples"] = torch.from_numpy(np.ascontiguousarray(u.real)).cuda().requires_grad_(True)
        state["target"] = torch.from_numpy(_unitary(seed, case["d"]).astype(H0.dtype)).cuda()
    return state


def run(state):
    if state["kind"] == "ensemble":
        state["ens"].set_samples(state["samples"])
        return np.concatenate([U.ravel() for U in state["ens"].run()])
    if state["kind"] == "host":
        return state["ctx"].equiprop(state["dt"], *state["samples"])
    if state["kind"] == "device":
        return state["ctx"].equiprop_device(state["dt"], state["samples"])
    u = state["samples"]
    U = propagate(state["ctx"], state["dt"], u)
    loss = fidelity_loss(U, state["target"])
    grad, = torch.autograd.grad(loss, u)
    return {"U": U.detach(), "loss": loss.detach(), "grad": grad}


# ------------------------------------------------------------------ the work

def _step_flops(d, Ke):
    """One step: its Hamiltonian from 1 + Ke matrices, an exponential to a
    degree of five or more (three complex products at least) and the product
    with what came before."""
    return 8.0 * Ke * d * d + 4 * 8.0 * d ** 3


def work(case):
    es = 8.0 if case["precision"] == "fp32" else 16.0
    if case["kind"] == "ensemble":
        n, pts, K = case["n"], 0.5 * (case["pts_min"] + case["pts_max"]), 2.5
        return dict(bytes=n * es * (K * pts + sum(p * (2 + K) * d * d for d, p in zip(ENS_DIMS, ENS_SHARE))),
                    flops=n * pts * sum(p * _step_flops(d, K) for d, p in zip(ENS_DIMS, ENS_SHARE)))
    d, K, P = case["d"], case["K"], case["steps"]
    Ke = 2 * K + K * (K - 1) // 2 if case["magnus"] else K
    samples = K * _points(case)
    got = dict(bytes=es * (samples + (2 + K) * d * d), flops=P * _step_flops(d, Ke))
    if case["kind"] == "grad":
        # Backward: the derivative of three products (two each), the seed
        # carried through the step, a trace with every expansion matrix.
        got["flops"] += P * (8 * 8.0 * d ** 3 + 8.0 * Ke * d * d)
        got["bytes"] += es / 2 * samples + es * d * d
    return got


# ------------------------------------------------------------------ 64 bits

def _stack(H0, H1, magnus):
    """[H0, H_k] and, for Magnus steps, [H0, H_k] and [H_j, H_i] (j < i)."""
    mats = [H0] + list(H1)
    if magnus:
        K = len(H1)
        mats += [H0 @ H - H @ H0 for H in H1]
        mats += [H1[j] @ H1[i] - H1[i] @ H1[j] for i in range(1, K) for j in range(i)]
    return torch.stack(mats)


def _weights(u, h, quadrature, magnus):
    """Weights (steps, 1 + Ke) of the stack from the complex samples (K, n)."""
    if quadrature == "simpson":
        a, b, c = u[:, 0:-2:2], u[:, 1:-1:2], u[:, 2::2]
        w = [(a + 4 * b + c) / 6]
        if magnus:
            K, f = u.shape[0], 1j * h / 12
            w.append(f * (c - a))
            w += [(f * (a[j] * c[i] - c[j] * a[i]))[None] for i in range(1, K) for j in range(i)]
        w = torch.cat(w)
    elif quadrature == "midpoint":
        w = 0.5 * (u[:, 1:] + u[:, :-1])
    else:
        w = u
    return torch.cat([torch.ones_like(w[:1]), w]).T


def _ordered(U):
    """Product of U (n, d, d), later factors on the left."""
    while U.shape[0] > 1:
        n = U.shape[0] // 2
        W = U[1:2 * n:2] @ U[0:2 * n:2]
        U = torch.cat([W, U[2 * n:]]) if U.shape[0] % 2 else W
    return U[0]


def _propagator(stack, w, h):
    """prod_j exp(-i h X_j), X_j = sum_m w_jm S_m: Taylor series to 2^-60."""
    d = stack.shape[1]
    x = h * float((w.detach().abs() @ stack.abs().sum(-1).amax(-1)[:, None].to(w.real.dtype)).max())
    n, term = 1, x
    while term > 2.0 ** -60:
        n += 1
        term *= x / n
    eye = torch.eye(d, dtype=stack.dtype, device=stack.device)
    slab, parts = max(1, (1 << 25) // (d * d)), []
    for s in range(0, w.shape[0], slab):
        A = (w[s:s + slab] @ stack.reshape(stack.shape[0], d * d)).reshape(-1, d, d) * (-1j * h)
        V = eye + A / n
        for k in range(n - 1, 0, -1):
            V = eye + (A @ V) / k
        parts.append(_ordered(V))
    return _ordered(torch.stack(parts))


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def on(a):
        return torch.from_numpy(np.asarray(a, dtype=np.complex128)).to(dev)

    if case["kind"] == "ensemble":
        Us = [_propagator(_stack(on(H0), on(H1), False), _weights(on(u), case["dt"], "none", False), case["dt"])
              for H0, H1, u in _ensemble_problems(case, seed)]
        return torch.cat([U.reshape(-1) for U in Us]).cpu().numpy()
    H0, H1, u = _problem(case, seed)
    h = case["dt"] * (2 if case["quadrature"] == "simpson" else 1)
    stack = _stack(on(H0), on(H1), case["magnus"])
    if case["kind"] != "grad":
        U = _propagator(stack, _weights(on(u), h, case["quadrature"], case["magnus"]), h)
        return U.cpu().numpy() if case["kind"] == "host" else U
    x = on(u).real.clone().requires_grad_(True)
    U = _propagator(stack, _weights(x.to(torch.complex128), h, case["quadrature"], case["magnus"]), h)
    V = on(_unitary(seed, case["d"]).astype(H0.dtype))
    loss = 1.0 - torch.trace(V.conj().T @ U).abs() ** 2 / case["d"] ** 2
    grad, = torch.autograd.grad(loss, x)
    return {"U": U.detach(), "loss": loss.detach(), "grad": grad}
