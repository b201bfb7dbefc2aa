"""Block factorisation (csrc/k_fact.cu) of systems whose form of the row workspaces
depends on the number of rows: small ones take the wide form at once, larger ones
start with the narrow one, which leaves room for more warps, and take the wide one
when too many rows overflow.  The factor does not depend on the schedule or on the
form: it agrees with the oracle's as block factors do (density to 1 %, and the
preconditioner to 2e-2: the SVDs of near-identity pivot blocks differ by rotations,
which move blocks across the thresholds), and more warps run where rows are short."""
import numpy as np
import pytest

import problems as P

pytestmark = pytest.mark.gpu


def _factor(ctx, nn, kind, tau):
    import bsg
    s = P.lame3d(nn, sigma=0.5, seed=3)
    u = s.upper() if kind == "ich2" else s
    p = bsg.default_param(ordtype=0, fcttyp=2, tau1=tau, tau2=tau, theta=0.1, memory=60.0)
    m = bsg.Matrix(ctx, u.n, u.ia, u.ja, u.a, 3, kind == "ich2")
    f = bsg.Factor(ctx, m, kind, p)
    return s, m, f, p, bsg.fact_stats()


@pytest.mark.parametrize("kind", ["ich2", "ilu2"])
def test_large_systems_of_short_rows_get_more_warps(ctx, kind):
    warps = {}
    for nn in (32, 33):  # 32768 and 35937 block rows
        s, m, f, p, st = _factor(ctx, nn, kind, 0.1)
        warps[nn] = st["warps"]
        assert st["big_rows"] == 0
        f.free()
        m.free()
    assert warps[33] > warps[32]


@pytest.mark.parametrize("nn,tau", [(32, 0.03), (33, 0.03), (33, 3e-4)])
def test_forms_agree_with_the_oracle(ctx, oracle, nn, tau):
    s, m, f, p, st = _factor(ctx, nn, "ich2", tau)
    u = s.upper()
    ia, ja, l, uu = f.export_block()
    o = oracle.ich2_block(u.ia, u.ja, u.a, 3, tau1=tau, tau2=tau, theta=0.1)
    assert abs(p.density - o[3][0]) <= 0.01 * o[3][0]
    x = np.random.default_rng(5).standard_normal(3 * s.n)
    y, z = (oracle.solve_u_block(a, b, v, 3, oracle.solve_l_block(a, b, v, 3, x)) for a, b, v in
            ((ia, ja, uu), (o[0], o[1], o[2])))
    assert np.linalg.norm(y - z) <= 2e-2 * np.linalg.norm(z)
    f.free()
    m.free()
