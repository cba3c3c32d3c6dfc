"""A capture after an ordinary call of the same size at another step length: where the
kernels of x = Hnorm h <= 1 keep buffers of their own, the captured call runs with
those that the ordinary call left.  The replay gives, to the bars of the contexts,
what a fresh context gives.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problem(precision, d, pts):
    import torch
    rng = np.random.default_rng((d, pts))
    ct = np.complex64 if precision == "fp32" else np.complex128

    def h():
        a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
        return ((a + a.conj().T) / (4 * np.sqrt(d))).astype(ct)

    H0, H1 = h(), [h(), h()]
    hn = sum(np.abs(m).sum(0).max() for m in (H0, *H1))
    return H0, H1, float(hn), torch.from_numpy(rng.uniform(-1.0, 1.0, (2, pts)).astype(ct)).cuda()


def replayed(call, out):
    import torch
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    got = out.clone()
    call()  # ordinary calls go on
    torch.cuda.synchronize()
    return got


@pytest.mark.parametrize("precision,d,pts,first,second", [
    ("fp32", 2, 300, 2.0, 0.1), ("fp32", 8, 5000, 2.0, 0.1), ("fp64", 3, 300, 2.0, 0.1), ("fp64", 8, 5000, 2.0, 0.1),
    ("fp32", 8, 5000, 0.1, 2.0), ("fp64", 4, 700, 0.1, 2.0), ("fp32", 27, 300, 2.0, 0.1), ("fp32", 64, 300, 2.0, 0.1),
    ("fp32", 96, 33, 2.0, 0.1), ("fp32", 200, 9, 2.0, 0.1), ("fp64", 24, 65, 2.0, 0.1), ("fp64", 24, 65, 0.1, 2.0)])
def test_equiprop(built_lib, precision, d, pts, first, second):
    import torch

    import parament_gb300 as parament
    H0, H1, hn, u = problem(precision, d, pts)
    with parament.Parament(precision) as ctx, parament.Parament(precision) as fresh:
        for c in (ctx, fresh):
            c.set_hamiltonian(H0, *H1)
        ref = fresh.equiprop_device(second / hn, u)
        out = torch.empty_like(ref)
        ctx.equiprop_device(first / hn, u, out=out)
        got = replayed(lambda: ctx.equiprop_device(second / hn, u, out=out), out)
        off = (torch.linalg.norm(got - ref) / torch.linalg.norm(ref)).item()
        assert off < (1e-5 if precision == "fp32" else 1e-10) * max(1.0, pts / 300)


@pytest.mark.parametrize("precision,d,first,second", [("fp32", 8, 2.0, 0.1), ("fp32", 32, 0.1, 2.0),
                                                      ("fp32", 40, 2.0, 0.1), ("fp64", 12, 0.1, 2.0),
                                                      ("fp64", 32, 2.0, 0.1)])
def test_gradients(built_lib, precision, d, first, second):
    import torch

    import parament_gb300 as parament
    H0, H1, hn, u = problem(precision, d, 3000)
    W = torch.eye(d, dtype=u.dtype, device="cuda")
    with parament.Parament(precision) as ctx, parament.Parament(precision) as fresh:
        for c in (ctx, fresh):
            c.set_hamiltonian(H0, *H1)
        ref = fresh.vjp_device(second / hn, u, W)
        out = torch.empty_like(ref)
        ctx.vjp_device(first / hn, u, W, grad=out)
        got = replayed(lambda: ctx.vjp_device(second / hn, u, W, grad=out), out)
        assert torch.equal(got, ref)


@pytest.mark.parametrize("precision,d,steps,fewer", [("fp64", 18, 900, 60), ("fp64", 8, 900, 5), ("fp64", 20, 400, 152),
                                                     ("fp32", 5, 900, 7), ("fp64", 40, 900, 60)])
def test_fewer_steps(built_lib, precision, d, steps, fewer):
    """A capture of fewer steps than the ordinary call had, by another kernel or not."""
    import torch

    import parament_gb300 as parament
    H0, H1, hn, u = problem(precision, d, steps)
    v = u[:, :fewer].contiguous()
    with parament.Parament(precision) as ctx, parament.Parament(precision) as fresh:
        for c in (ctx, fresh):
            c.set_hamiltonian(H0, *H1)
        ref = fresh.equiprop_device(0.005 / hn, v)
        out = torch.empty_like(ref)
        ctx.equiprop_device(0.005 / hn, u, out=out)
        assert torch.equal(replayed(lambda: ctx.equiprop_device(0.005 / hn, v, out=out), out), ref)
