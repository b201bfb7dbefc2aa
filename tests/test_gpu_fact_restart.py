"""When a factorisation starts again with wider row workspaces (csrc/k_fact.cu): not
for rows that the matrix itself makes long, which the wider ones need not take
either.  Such rows early in the matrix leave the factor with the warps of one
without them, and with the oracle's bits."""
import numpy as np
import pytest
import scipy.sparse as sp

import problems as P

pytestmark = pytest.mark.gpu


def _system(nlong):
    """A 2-D grid of 20000 rows, nlong rows after the 600th with 350 earlier neighbours."""
    s = P.heat3d(200, 100, 1, sigma=1.0, seed=4)
    A = sp.csr_matrix((s.a, s.ja, s.ia), shape=(s.n, s.n))
    T = sp.triu(A, 1).tocoo()
    rng = np.random.default_rng(nlong)
    rows = np.repeat(600 + 2 * np.arange(nlong), 350)
    cols = np.concatenate([rng.choice(600, 350, replace=False) for _ in range(nlong)]) if nlong else rows
    B = sp.coo_matrix((np.r_[T.data, np.full(len(rows), -0.01)], (np.r_[T.row, cols], np.r_[T.col, rows])),
                      shape=(s.n, s.n)).tocsr()
    d = np.asarray(abs(B).sum(1)).ravel() + np.asarray(abs(B).sum(0)).ravel() + 1.0
    return sp.csr_matrix(sp.triu(B, 1) + sp.diags(d)).sorted_indices()


def test_rows_that_the_matrix_makes_long(ctx, oracle):
    import bsg
    warps = []
    for nlong in (0, 200):
        A = _system(nlong)
        m = bsg.Matrix(ctx, A.shape[0], A.indptr, A.indices, A.data, 1, True)
        p = bsg.default_param(ordtype=0, fcttyp=2, tau1=1e-2, tau2=1e-2, memory=60.0)
        f = bsg.Factor(ctx, m, "ich2", p)
        warps.append(bsg.fact_stats()["warps"])
        giu, gju, _, gu = f.export()
        iu, ju, uu, _, _ = oracle.fact(0, A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, tau1=1e-2,
                                       tau2=1e-2)
        assert np.array_equal(giu, iu) and np.array_equal(gju, ju) and np.array_equal(gu, uu)
        f.free()
        m.free()
    assert warps[0] == warps[1]
