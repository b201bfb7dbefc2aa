"""The time limit of an exact solve (bsg_set_spin_limit_ns) counts from the last
row solved, not from the launch: on a chain the last block of rows waits for all
the blocks before it, several times the limit here, and the solve still ends with
the bits of an unhurried one, which are held to the backward error of substitution,
(k + 4) 2^-53 for rows of k entries (Higham, Accuracy and Stability of Numerical
Algorithms, theorem 8.5).  (test_gpu_failure.py has the limit run out.)"""
import numpy as np
import pytest
import scipy.sparse as sp

import problems as P

pytestmark = pytest.mark.gpu

DEFAULT_NS = 2_000_000_000
SHORT_NS = 20_000_000  # a link takes less than a microsecond, the chain more than 60 ms


@pytest.mark.parametrize("lower", [1, 0])
def test_progress_starts_the_limit_again(ctx, lower):
    import bsg
    import torch
    s = P.heat3d(400_000, 1, 1, sigma=1.0, seed=5)
    m = bsg.Matrix.from_system(ctx, s, symm_upper=True)
    f = bsg.Factor(ctx, m, "ich2", bsg.default_param(ordtype=0, fcttyp=1))
    solve = f.solve_l if lower else f.solve_u
    x = torch.as_tensor(np.random.default_rng(1).standard_normal(s.n), device="cuda")
    y = torch.empty_like(x)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    ev[0].record()
    solve(x, y, mode=0)
    ev[1].record()
    ctx.sync()
    assert ev[0].elapsed_time(ev[1]) * 1e6 > 2 * SHORT_NS  # the wait would run out
    z = torch.empty_like(x)
    try:
        assert bsg.lib().bsg_set_spin_limit_ns(ctx.h, SHORT_NS) == bsg.OK
        solve(x, z, mode=0)
        ctx.sync()
    finally:
        assert bsg.lib().bsg_set_spin_limit_ns(ctx.h, DEFAULT_NS) == bsg.OK
    assert torch.equal(y, z)
    # componentwise backward error of substitution, rows of two entries
    iu, ju, _, u = f.export()
    first = np.zeros(len(ju), bool)
    first[iu[:-1]] = True
    S = sp.csr_matrix((np.where(first, 0.0, u), ju, iu), shape=(s.n, s.n))
    S = S.T.tocsr() if lower else S
    got, rhs = z.cpu().numpy(), x.cpu().numpy()
    r = S @ got + got / u[first] - rhs
    assert np.all(abs(r) <= 6 * 2.0 ** -53 * (abs(S) @ abs(got) + abs(got / u[first]) + abs(rhs)))
    f.free()
    m.free()
