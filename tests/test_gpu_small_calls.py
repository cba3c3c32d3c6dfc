"""Host-buffer calls of up to 16 KB of samples and of result go through pinned memory
that the kernels reach directly; larger ones are copied.  Both sides of either limit
give, bit for bit, what the device entry point gives, in every form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,form,d,pts", [
    ("fp32", "plain", 4, 2048), ("fp32", "plain", 4, 2049), ("fp32", "plain", 45, 60), ("fp32", "plain", 46, 60),
    ("fp32", "split", 12, 2048), ("fp32", "split", 12, 2049), ("fp64", "plain", 3, 1024), ("fp64", "plain", 3, 1025),
    ("fp64", "plain", 12, 300), ("fp64", "plain", 32, 40), ("fp64", "plain", 33, 40), ("fp64", "plain", 2, 1)])
def test_staged_calls_match_the_device_entry_point(built_lib, precision, form, d, pts):
    import torch

    import parament_gb300 as parament
    rng = np.random.default_rng((d, pts))
    ct = np.complex64 if precision == "fp32" else np.complex128
    a = rng.standard_normal((2, d, d)) + 1j * rng.standard_normal((2, d, d))
    H = ((a + a.conj().transpose(0, 2, 1)) / (4 * np.sqrt(d))).astype(ct)
    u = rng.standard_normal((1, pts)).astype(ct)
    with parament.Parament(precision) as ctx:
        if form != "plain":
            ctx.set_precision_mode(form)
        ctx.set_hamiltonian(H[0], H[1])
        for dt in (1e-3, 0.0, 2e-3):
            U = ctx.equiprop(dt, *u)
            D = ctx.equiprop_device(dt, torch.from_numpy(u).cuda())
            ctx.synchronize()
            assert np.array_equal(U, D.cpu().numpy())
