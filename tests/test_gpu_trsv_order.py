"""Exact solves (csrc/k_trsv.cu) of factors whose wavefronts do not suit blocks of
rows: graphs with links in a window, without locality, and permuted grids, above
the size where solves may go by rows in level order, and controls just below it and
with locality.  The bound is test_gpu_trsv.py's componentwise backward error, (k + 4)
2^-53 for rows of k entries.  bsg_launch_count tells which order was chosen: the one
by rows sorts again, one launch of the library more."""
import numpy as np
import pytest
import scipy.sparse as sp

import problems as P

pytestmark = pytest.mark.gpu


def _graph(n, deg, window, seed=1):
    rng = np.random.default_rng(seed)
    r = rng.integers(0, n, deg * n)
    c = rng.integers(0, n, deg * n) if window is None else r + rng.integers(-window, window + 1, deg * n)
    ok = (c >= 0) & (c < n) & (c != r)
    A = sp.coo_matrix((-rng.random(ok.sum()), (r[ok], c[ok])), shape=(n, n)).tocsr()
    A = A + A.T
    return sp.csr_matrix(A + sp.diags(1.0 - np.asarray(A.sum(1)).ravel()))


def _grid(dims, permute):
    s = P.heat3d(*dims, sigma=1.0, seed=3)
    A = sp.csr_matrix((s.a, s.ja, s.ia), shape=(s.n, s.n))
    p = np.random.default_rng(0).permutation(s.n) if permute else np.arange(s.n)
    return sp.csr_matrix(A[p][:, p])


IC0 = dict(fcttyp=1)
IC2 = dict(fcttyp=2, tau1=1e-2, tau2=1e-2, memory=40.0)
CASES = {  # matrix, factor, solved by rows
    "window": (lambda: _graph(250000, 3, 20000), IC0, True),
    "eight neighbours": (lambda: _graph(200000, 8, None), IC0, True),
    "permuted grid": (lambda: _grid((64, 64, 64), True), IC2, True),
    "just below the size": (lambda: _graph(49999, 8, None), IC0, False),
    "few links": (lambda: _graph(150000, 1, 10000), IC0, False),
    "natural grid": (lambda: _grid((60, 50, 40), False), IC2, False),
}


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_solve_order(ctx, name, fp32):
    import bsg
    import torch
    make, par, by_rows = CASES[name]
    A = sp.triu(make()).tocsr().sorted_indices()
    n = A.shape[0]
    m = bsg.Matrix(ctx, n, A.indptr, A.indices, A.data, 1, True)
    f = bsg.Factor(ctx, m, "ich2", bsg.default_param(ordtype=0, **par))
    iu, ju, _, u = f.export()
    first = np.zeros(len(ju), bool)
    first[iu[:-1]] = True
    if fp32:
        f.to_fp32()
        u = np.where(first, u, u.astype(np.float32))
    U = sp.csr_matrix((np.where(first, 0.0, u), ju, iu), shape=(n, n))
    x = np.random.default_rng(n).standard_normal(n)
    d_x, d_y = torch.as_tensor(x, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    for solve, S in ((f.solve_l, U.T.tocsr()), (f.solve_u, U)):
        solve(d_x, d_y, mode=0)
        y = d_y.cpu().numpy()
        k = int(np.diff(S.indptr).max())
        r = S @ y + y / u[first] - x
        assert np.all(abs(r) <= (k + 4) * 2.0 ** -53 * (abs(S) @ abs(y) + abs(y / u[first]) + abs(x)))
    f.free()
    m.free()


@pytest.mark.parametrize("name", [k for k in sorted(CASES) if CASES[k][1] is IC0])
def test_order_that_is_taken(ctx, name):
    import bsg

    def launches(A):
        A = sp.triu(A).tocsr().sorted_indices()
        m = bsg.Matrix(ctx, A.shape[0], A.indptr, A.indices, A.data, 1, True)
        before = bsg.lib().bsg_launch_count()
        f = bsg.Factor(ctx, m, "ich2", bsg.default_param(ordtype=0, **IC0))
        count = bsg.lib().bsg_launch_count() - before
        f.free()
        m.free()
        return count

    make, _, by_rows = CASES[name]
    A = make()
    n = A.shape[0]
    chain = sp.diags([np.full(n - 1, -1.0), np.full(n, 3.0), np.full(n - 1, -1.0)], [-1, 0, 1])
    assert launches(A) - launches(chain) == int(by_rows)
