"""Device-buffer calls captured in a CUDA graph: each form's first captured calls
after an ordinary one, two in one capture, replayed on new samples.  A replay runs
the kernels of the ordinary call on the same buffers, so the results are the same
bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,form,d,pts", [
    ("fp64", "plain", 3, 300), ("fp64", "plain", 12, 200), ("fp64", "plain", 24, 65), ("fp64", "magnus", 64, 65),
    ("fp64", "plain", 96, 33), ("fp32", "plain", 4, 300), ("fp32", "plain", 27, 300), ("fp32", "plain", 64, 200),
    ("fp32", "midpoint", 128, 33), ("fp32", "magnus_split", 96, 33)])
def test_capture_and_replay(built_lib, precision, form, d, pts):
    import torch
    import parament_gb300 as parament
    from parament_gb300.workloads import hermitian
    rng = np.random.default_rng(d)
    H0 = hermitian(rng, d, 1.0)
    H1 = np.stack([hermitian(rng, d, 1.0) for _ in range(2)])
    ct = torch.complex64 if precision == "fp32" else torch.complex128
    u = [torch.from_numpy(rng.normal(size=(2, pts))).to("cuda", ct) for _ in range(2)]
    with parament.Parament(precision) as ctx:
        if form.endswith("_split"):
            ctx.set_precision_mode("split")
        ctx.set_hamiltonian(H0, *H1, use_magnus=form.startswith("magnus"),
                            quadrature_mode={"plain": "none", "midpoint": "midpoint"}.get(form, "simpson"))
        ref = [ctx.equiprop_device(1e-3, x).clone() for x in u]
        x, y = u[0].clone(), u[1].clone()
        a, b = torch.empty_like(ref[0]), torch.empty_like(ref[0])
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ctx.equiprop_device(1e-3, x, out=a)
            ctx.equiprop_device(1e-3, y, out=b)
        for p, q in ((0, 1), (1, 0)):
            x.copy_(u[p])
            y.copy_(u[q])
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(a, ref[p]) and torch.equal(b, ref[q])
        assert torch.equal(ctx.equiprop_device(1e-3, u[0]), ref[0])
        del g
