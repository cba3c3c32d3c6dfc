"""Reports of bounded waits that gave up, through every way a call is made: host
buffers, device buffers, a CUDA graph's replays.  The give-up is made on the host
(PARAMENT_FAIL_WAIT_AFTER): no kernel waits in vain.  And a context synchronises after
a capture, whether its kernels have bounded waits or not.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import numpy as np, torch, parament_gb300 as p
how = "%s"
rng = np.random.default_rng(1)
a = rng.standard_normal((2, %d, %d)); H = (a + a.transpose(0, 2, 1)) / 10
u = rng.standard_normal((1, 400))
x = torch.from_numpy(u + 0j).cuda()

def report(f):
    try:
        f()
        print("fine")
    except RuntimeError as e:
        print("gave up" if "1010" in str(e) else e)

with p.Parament("fp64") as ctx:
    ctx.set_hamiltonian(H[0], H[1])
    if how == "host":
        report(lambda: ctx.equiprop(1e-3, *u))
        report(lambda: ctx.equiprop(1e-3, *u))
    elif how == "device":
        ctx.equiprop_device(1e-3, x)
        report(ctx.synchronize)
        report(ctx.synchronize)
    elif how == "next call":
        ctx.equiprop_device(1e-3, x)
        torch.cuda.synchronize()
        report(lambda: ctx.equiprop_device(1e-3, x))
        report(lambda: ctx.equiprop_device(1e-3, x))
    else:
        out = ctx.equiprop_device(1e-3, x)
        ctx.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ctx.equiprop_device(1e-3, x, out=out)
        report(ctx.synchronize)
        g.replay()
        torch.cuda.synchronize()
        report(ctx.synchronize)
        report(ctx.synchronize)
"""


def run(how, d, after):
    env = dict(os.environ)
    env.pop("PARAMENT_FAIL_WAIT_AFTER", None)
    if after is not None:
        env["PARAMENT_FAIL_WAIT_AFTER"] = str(after)
    r = subprocess.run([sys.executable, "-c", PROGRAM % (how, d, d)], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    return r.stdout.split("\n")[:-1]


@pytest.mark.parametrize("how,after,lines", [
    ("host", 0, ["gave up", "fine"]), ("device", 0, ["gave up", "fine"]), ("next call", 0, ["gave up", "fine"]),
    ("replay", 1, ["fine", "gave up", "fine"]), ("replay", None, ["fine", "fine", "fine"])])
def test_reports(built_lib, how, after, lines):
    assert run(how, 64, after) == lines


def test_a_context_without_waits(built_lib):
    assert run("replay", 6, None) == ["fine", "fine", "fine"]


def test_gradients_and_synchronize(built_lib):
    import torch

    import parament_gb300 as parament
    rng = np.random.default_rng(3)
    a = rng.standard_normal((2, 12, 12))
    H = (a + a.transpose(0, 2, 1)) / 10
    u = torch.from_numpy(rng.standard_normal((1, 50)) + 0j).cuda()
    W = torch.eye(12, dtype=u.dtype, device="cuda")
    with parament.Parament("fp64") as ctx:
        ctx.set_hamiltonian(H[0], H[1])
        ref = ctx.vjp_device(1e-3, u, W)
        out = torch.empty_like(ref)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ctx.vjp_device(1e-3, u, W, grad=out)
        ctx.synchronize()
        g.replay()
        torch.cuda.synchronize()
        ctx.synchronize()
        assert torch.equal(out, ref)
