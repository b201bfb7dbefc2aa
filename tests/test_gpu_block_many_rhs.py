"""Block sweeps of more vectors than one pass takes (groups of 8): every vector,
the one of a group of its own among them, gets the bits of its own solve."""
import pytest

import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr", [7, 8, 9, 10, 16, 17])
@pytest.mark.parametrize("precision", [0, 1])
def test_vectors_beyond_a_group_of_eight(ctx, nr, precision):
    import bsg
    import torch
    s = P.lame3d(5, sigma=0.5, seed=3)
    m = bsg.Matrix(ctx, s.n, s.ia, s.ja, s.a, 3, False)
    f = bsg.Factor(ctx, m, "ilu2", bsg.default_param(ordtype=0, fcttyp=2, tau1=1e-3, tau2=1e-3, memory=40.0,
                                                     precision=precision))
    g = torch.Generator(device="cuda").manual_seed(nr)
    X = torch.randn((nr, 3 * s.n), generator=g, dtype=torch.float64, device="cuda")
    Y, y = torch.empty_like(X), torch.empty_like(X[0])
    for sweeps in (2, 3, 6):
        f.solve_multi(1, X, Y, 1, sweeps)
        for q in range(nr):
            f.solve_l(X[q].contiguous(), y, mode=1, nsweeps=sweeps)
            assert torch.equal(y, Y[q]), (sweeps, q)
    f.free()
    m.free()
