"""Block sweeps with several lanes a block row (csrc/k_bsell.cu, small systems)
against plain block arithmetic around the sizes where lanes run out, and against
the lane-a-row kernel of larger systems: below 24000 block rows several FP64
vectors share lanes while a single one (above 12000 rows) does not, and both must
give a vector the same bits."""
import numpy as np
import pytest
import scipy.sparse as sp

import problems as P

pytestmark = pytest.mark.gpu


def _parts(f):
    """Strict part and diagonal blocks of the upper block factor: (N, D)."""
    ia, ja, _, u = f.export_block()
    nb = len(ia) - 1
    blocks = u.reshape(-1, 3, 3).transpose(0, 2, 1)
    first = np.zeros(len(ja), bool)
    first[ia[:-1]] = True
    rows = np.repeat(np.arange(nb), np.diff(ia))
    N = sp.bsr_matrix((blocks[~first], ja[~first], np.concatenate([[0], np.cumsum(np.diff(ia) - 1)])),
                      shape=(3 * nb, 3 * nb)).tocsr()
    return N, blocks[first], rows


@pytest.mark.parametrize("nn", [2, 3, 5])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_small_block_sweeps(ctx, nn, periodic, precision):
    import bsg
    import torch
    if periodic and nn < 3:
        pytest.skip("a periodic cell needs three nodes a side")
    s = P.lame_periodic(nn, rmin=0.6, rmax=1.0) if periodic else P.lame3d(nn, sigma=0.5, seed=3)
    u = s.upper()
    m = bsg.Matrix(ctx, u.n, u.ia, u.ja, u.a, 3, True)
    f = bsg.Factor(ctx, m, "ich2", bsg.default_param(ordtype=0, fcttyp=2, tau1=1e-3, tau2=1e-3, memory=40.0))
    N, D, _ = _parts(f)
    if precision:
        f.to_fp32()
        N.data = N.data.astype(np.float32).astype(np.float64)
    rng = np.random.default_rng(nn)
    for nr in (1, 2, 3, 4, 5, 6, 8, 9):
        X = rng.standard_normal((nr, 3 * s.n))
        Y = torch.empty((nr, 3 * s.n), dtype=torch.float64, device="cuda")
        f.solve_multi(0, torch.as_tensor(X, device="cuda"), Y, 1, 4)
        got = Y.cpu().numpy()
        for q in range(nr):
            dot = lambda t: np.einsum("irc,ic->ir", D, t.reshape(-1, 3)).reshape(-1)  # noqa: E731
            y, scale = dot(X[q]), 0.0
            for _ in range(3):
                scale = abs(N) @ abs(y) + abs(X[q])
                y = dot(X[q] - N @ y)
            # a row's sum of k products and the 3 x 3 product, each rounding
            # once, three sweeps deep, against the size of what was added
            k = 3 * int(np.diff(N.indptr).max() + 8)
            lim = np.einsum("irc,ic->ir", abs(D), scale.reshape(-1, 3)).max()
            assert np.abs(got[q] - y).max() <= k * 2.0 ** -53 * max(lim, np.abs(y).max()) * 3, (nr, q)
    f.free()
    m.free()


def test_shared_lanes_give_the_bits_of_a_lane_a_row(ctx):
    import bsg
    import torch
    s = P.lame3d(27, sigma=0.5, seed=3)
    assert 12000 < s.n <= 24000
    m = bsg.Matrix(ctx, s.n, s.ia, s.ja, s.a, 3, False)
    f = bsg.Factor(ctx, m, "ilu2", bsg.default_param(ordtype=0, fcttyp=2, tau1=1e-2, tau2=1e-2, memory=20.0))
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn((6, 3 * s.n), generator=g, dtype=torch.float64, device="cuda")
    Y, y = torch.empty_like(X), torch.empty_like(X[0])
    for lower in (1, 0):
        f.solve_multi(lower, X, Y, 1, 4)
        for q in range(6):
            (f.solve_l if lower else f.solve_u)(X[q].contiguous(), y, mode=1, nsweeps=4)
            assert torch.equal(y, Y[q])
    f.free()
    m.free()
