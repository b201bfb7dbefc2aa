"""Exact triangular solves (csrc/k_trsv.cu) where their block layout can go
wrong: row counts around a block of 256 rows, links that cross blocks (a chain
runs through all of them), rows longer than the 64 entries a warp holds at once,
FP32 factor values, the transposed forms, and more blocks than one launch takes.

The solution y of D^{-1} y + N y = x is held to the componentwise backward error of
substitution with rows of k entries, (k + 4) 2^-53, for the rows' absolute sums
(Higham, Accuracy and Stability of Numerical Algorithms, theorem 8.5), so the
bound needs no condition number.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import problems as P

pytestmark = pytest.mark.gpu


def _system(kind, n):
    """Upper CSR (diagonal first) of a diagonally dominant matrix."""
    if kind == "chain":
        U = sp.diags([np.full(n - 1, -1.0)], [1], shape=(n, n))
    elif kind == "arrow":  # the last row and column are full
        U = sp.csr_matrix((np.full(n - 1, -0.5), (np.arange(n - 1), np.full(n - 1, n - 1))), shape=(n, n))
        U = U + sp.diags([np.full(n - 2, -1.0)], [2], shape=(n, n))
    else:  # 2-D grid as square as it goes
        m = int(np.sqrt(n))
        U = sp.diags([np.full(n - 1, -1.0), np.full(n - m, -1.0)], [1, m], shape=(n, n))
    U = sp.csr_matrix(U)
    d = np.asarray(abs(U).sum(1)).ravel() + np.asarray(abs(U).sum(0)).ravel() + 1.0
    return sp.csr_matrix(sp.triu(U, 1) + sp.diags(d)).sorted_indices()


def _check(S, dinv, x, y, k):
    """Componentwise backward error of (strict part S + diag(1 / dinv)) y = x."""
    r = S @ y + y / dinv - x
    scale = abs(S) @ abs(y) + abs(y / dinv) + abs(x)
    assert np.all(np.isfinite(y))
    assert np.all(abs(r) <= (k + 4) * 2.0 ** -53 * scale)


def _solve_and_check(ctx, A, param, kind="ich2", fp32=False, transposed=False):
    import bsg
    import torch
    n = A.shape[0]
    if kind == "ich2":
        m = bsg.Matrix(ctx, n, A.indptr, A.indices, A.data, 1, True)
    else:  # nonsymmetric values on the full pattern, diagonal first
        L = sp.tril(A.T, -1).tocsr() * 0.7
        rows = [np.concatenate([[i], L.indices[L.indptr[i]:L.indptr[i + 1]],
                                A.indices[A.indptr[i] + 1:A.indptr[i + 1]]]) for i in range(n)]
        vals = [np.concatenate([[A.data[A.indptr[i]]], L.data[L.indptr[i]:L.indptr[i + 1]],
                                A.data[A.indptr[i] + 1:A.indptr[i + 1]]]) for i in range(n)]
        ia = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
        m = bsg.Matrix(ctx, n, ia, np.concatenate(rows), np.concatenate(vals), 1, False)
    f = bsg.Factor(ctx, m, kind, param)
    iu, ju, l, u = f.export()
    first = np.zeros(len(ju), bool)
    first[iu[:-1]] = True
    if fp32:
        f.to_fp32()
        l, u = (np.where(first, v, v.astype(np.float32)) for v in (l, u))
    U = sp.csr_matrix((np.where(first, 0.0, u), ju, iu), shape=(n, n))
    L = sp.csr_matrix((np.where(first, 0.0, l), ju, iu), shape=(n, n))  # rows of L^T
    k = int(np.diff(iu).max())
    kt = int(np.bincount(ju, minlength=n).max())
    x = np.random.default_rng(n).standard_normal(n)
    d_x, d_y = torch.as_tensor(x, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    runs = [(f.solve_l, L.T.tocsr(), l[first], kt), (f.solve_u, U, u[first], k)]
    if transposed:
        runs += [(f.solve_ut, U.T.tocsr(), u[first], kt), (f.solve_lt, L, l[first], k)]
    for solve, S, dinv, kk in runs:
        solve(d_x, d_y, mode=0)
        _check(S, dinv, x, d_y.cpu().numpy(), kk)
    f.free()
    m.free()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 511, 513, 2049])
@pytest.mark.parametrize("kind", ["chain", "arrow", "grid"])
def test_exact_solves_around_block_edges(ctx, kind, n):
    import bsg
    if n < 4 and kind != "chain":
        pytest.skip("no such pattern")
    A = _system(kind, n)
    _solve_and_check(ctx, A, bsg.default_param(ordtype=0, fcttyp=1))
    _solve_and_check(ctx, A, bsg.default_param(ordtype=0, fcttyp=1), fp32=True)


def test_exact_solves_transposed(ctx):
    import bsg
    p = bsg.default_param(ordtype=0, fcttyp=2, tau1=1e-3, tau2=1e-3, memory=40.0)
    _solve_and_check(ctx, _system("grid", 700), p, kind="ilu2", transposed=True)
    _solve_and_check(ctx, _system("grid", 700), p, kind="ilu2", fp32=True, transposed=True)


def test_exact_solves_of_several_launches(ctx):
    """More rows than 148 blocks of 28000 hold."""
    import bsg
    s = P.heat3d(2060, 2060, 1, sigma=0.5, seed=1).upper()
    A = sp.csr_matrix((s.a, s.ja, s.ia), shape=(s.n, s.n))
    _solve_and_check(ctx, A, bsg.default_param(ordtype=0, fcttyp=1))
