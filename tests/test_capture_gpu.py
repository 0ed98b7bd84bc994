"""An operator's first application inside the caller's stream capture: nothing that a
capture refuses is left to the launch.  In a process of its own, where no kernel has run."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import numpy as np, torch
from dmrgcc_b200 import capi
ctx = capi.Context(0)
stream = torch.cuda.ExternalStream(ctx.stream)
rng = np.random.default_rng(2)
up = lambda *s: capi.DeviceArray.from_host(ctx, rng.standard_normal(s))
m, n, bond = 33, 40, 2
z = 2 if KIND[0] == "z" else 1
W = rng.standard_normal((bond, bond, 1, 1)) + 1j * rng.standard_normal((bond, bond, 1, 1)) * (z - 1)
site = capi.SiteProblem(1, 1, np.zeros((1, 1)), capi.BlockSpec([0], [0], [m], [n]), W.real)
L, R = ([capi.BlockSpec([0], [0], [k], [k])] * bond for k in (m, n))
psi, dl, dr = up(z * m, n), up(bond, z * m, m), up(bond, z * n, n)
if KIND.endswith("env"):
    op, out = capi.Env(ctx, 0, site, L, Wc=W if z == 2 else None), up(bond, z * n, n)
    apply = lambda: op.apply(psi, dl, out)
else:
    op, out = capi.ZHeff(ctx, site, L, R, W) if z == 2 else capi.Heff(ctx, site, L, R), up(z * m, n)
    op.set_env(dl, dr)
    apply = lambda: op.apply(psi, out)
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=stream):
    apply()
out.zero()
with torch.cuda.stream(stream):
    graph.replay()
ctx.sync()
got = out.download()
apply()
ctx.sync()
assert np.any(got) and np.array_equal(got, out.download())
print("same")
"""


@pytest.mark.parametrize("kind", ["heff", "zheff", "env", "zenv"])
def test_first_application_in_a_capture(kind):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", f"KIND = {kind!r}" + PROGRAM], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]
