"""Block sweeps on both sides of the lines between lanes that share a block row and
a lane a row (csrc/k_bsell.cu: 12000 and 24000 block rows in FP64, 40000 in FP32).
A system with rows of its own behind it, to beyond the last line, has the same
factor rows and must get the same bits from the other kernel, with rows of more than
64 and of more than 1024 blocks, which whole warps and blocks take, among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BEYOND = 40008


def _matrix(ctx, nb, long_rows, total):
    """Upper blocks, diagonal first: neighbours i + 1 and i + 37, and the last rows
    as neighbours of as many rows before them as long_rows says; then single rows."""
    import bsg
    rng = np.random.default_rng(nb)
    rows = [[i, *(j for j in (i + 1, i + 37) if j < nb - len(long_rows))] for i in range(nb)]
    for q, k in enumerate(long_rows):
        j = nb - len(long_rows) + q
        for i in rng.choice(nb - len(long_rows), k, replace=False):
            rows[i].append(j)
    rows = [[i, *sorted(r[1:])] for i, r in enumerate(rows)]
    ia = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    a = rng.standard_normal((ia[-1], 9)) * 0.05
    a[ia[:-1]] = (np.eye(3) * 4.0).reshape(-1)
    extra = total - nb
    ia = np.concatenate([ia, ia[-1] + np.arange(1, extra + 1)])
    ja = np.concatenate([np.concatenate(rows), np.arange(nb, total)]).astype(np.int32)
    a = np.concatenate([a, np.tile(np.eye(3).reshape(-1), (extra, 1))])
    m = bsg.Matrix(ctx, total, ia, ja, a.ravel(), 3, True)
    p = bsg.default_param(ordtype=0, fcttyp=2, tau1=1e-6, tau2=1e-6, memory=60.0)
    return m, bsg.Factor(ctx, m, "ich2", p)


@pytest.mark.parametrize("nb,long_rows", [(1500, (1490, 1100, 200, 65)), (9000, ()), (9003, (700,))])
def test_both_kernels_give_the_same_bits(ctx, nb, long_rows):
    import torch
    small, large = (_matrix(ctx, nb, long_rows, t) for t in (nb, BEYOND))
    (ia, ja, _, u), (ib, jb, _, v) = (f.export_block() for _, f in (small, large))
    assert np.array_equal(ia, ib[:nb + 1]) and np.array_equal(ja, jb[:ia[-1]]) and np.array_equal(u, v[:len(u)])
    if long_rows:
        assert np.bincount(ja).max() > long_rows[0]
    for fp32 in (False, True):
        if fp32:
            small[1].to_fp32()
            large[1].to_fp32()
        for nr in (1, 2, 5, 6, 8, 9):
            X = torch.randn((nr, 3 * BEYOND), generator=torch.Generator(device="cuda").manual_seed(nr),
                            dtype=torch.float64, device="cuda")
            Xs, Y = X[:, :3 * nb].contiguous(), torch.empty_like(X)
            Ys = torch.empty_like(Xs)
            for lower in (1, 0):
                small[1].solve_multi(lower, Xs, Ys, 1, 4)
                large[1].solve_multi(lower, X, Y, 1, 4)
                assert torch.equal(Ys, Y[:, :3 * nb]), (fp32, nr, lower)
    for m, f in (small, large):
        f.free()
        m.free()
