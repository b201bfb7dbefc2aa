"""Exact solves on a part of the GPU: fewer SMs than the solve has blocks of rows.
Blocks are claimed in solve order, so a solve needs no number of CTAs resident at
once.  A child process gives the library a stream of a green context (a partition
of the SMs that ends with its process) and compares with the whole GPU, bit for
bit: a 3-D operator whose blocks follow one another and a chain through all."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys
import numpy as np
import torch
import bsg
import problems as P

part = torch.cuda.green_contexts.GreenContext.create(num_sms=int(sys.argv[1]), device_id=0)
stream = part.Stream()
whole = bsg.Context(0)
some = bsg.Context(0, stream.cuda_stream)
for dims, fcttyp in (((47, 40, 33), 2), ((60000, 1, 1), 1), ((3, 2, 1), 2)):
    s = P.heat3d(*dims, sigma=1.0, seed=3)
    p = bsg.default_param(ordtype=0, fcttyp=fcttyp, tau1=1e-3, tau2=1e-3, memory=40.0)
    x = torch.as_tensor(np.random.default_rng(2).standard_normal(s.n), device="cuda")
    out = []
    torch.cuda.synchronize()
    for c in (whole, some):
        m = bsg.Matrix.from_system(c, s, symm_upper=True)
        f = bsg.Factor(c, m, "ich2", p)
        y, z = torch.empty_like(x), torch.empty_like(x)
        torch.cuda.synchronize()
        f.solve_l(x, y, mode=0)
        f.solve_u(y, z, mode=0)
        c.sync()
        out.append((y.cpu(), z.cpu()))
        f.free()
        m.free()
    assert all(torch.equal(a, b) for a, b in zip(*out)), dims
print("same", flush=True)
"""


@pytest.mark.parametrize("sms", [8, 72])
def test_solve_on_a_part_of_the_gpu(sms):
    import torch
    if not hasattr(torch.cuda, "green_contexts"):
        pytest.skip("no green contexts in this PyTorch")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    path = os.pathsep.join([os.path.join(root, "bcm-problems_b200"), os.environ.get("PYTHONPATH", "")])
    r = subprocess.run([sys.executable, "-c", CHILD, str(sms)], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": path})
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
