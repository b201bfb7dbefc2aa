"""Row workspaces of the factorisation (csrc/k_fact.cu).  Factors whose rows do
not fit the usual shared workspace start again with the wide one: bit for bit
the oracle's.  Block rows keep up to 512 columns and members: a block factor with
rows of more than 256 agrees with the oracle's as the shorter ones do (the SVDs of
near-identity pivot blocks differ by rotations, which move blocks across the
thresholds: density to 1 %, preconditioner to 2e-2)."""
import numpy as np
import pytest

import problems as P

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("kind", ["ich2", "ilu2"])
@pytest.mark.parametrize("dims,sigma,tau,wide", [
    ((18, 18, 18), 1.0, 1e-4, True), ((16, 22, 18), 0.5, 1e-4, True), ((20, 20, 20), 1.0, 1e-3, False)])
def test_wide_factor_equals_oracle(ctx, oracle, dims, sigma, tau, wide, kind):
    import bsg
    s = P.heat3d(*dims, sigma=sigma, seed=3)
    u = s.upper()
    p = bsg.default_param(ordtype=0, fcttyp=2, tau1=tau, tau2=tau, memory=100.0)
    m = bsg.Matrix.from_system(ctx, s, symm_upper=True)
    f = bsg.Factor(ctx, m, kind, p)
    assert (bsg.fact_stats()["warps"] == 148 * 3 * 2) == wide
    giu, gju, gl, gu = f.export()
    iu, ju, lv, uv, _ = oracle.fact(0 if kind == "ich2" else 1, u.ia, u.ja, u.a, tau1=tau, tau2=tau)
    assert np.array_equal(giu, iu) and np.array_equal(gju, ju)
    assert np.array_equal(gl, lv) and np.array_equal(gu, uv)
    f.free()
    m.free()


def test_block_rows_of_more_than_256_columns(ctx, oracle):
    import bsg
    s = P.lame_periodic(9, rmin=1.5, rmax=2.5, seed=42)
    u = s.upper()
    p = bsg.default_param(ordtype=0, fcttyp=2, tau1=3e-4, tau2=3e-4, theta=0.1, memory=60.0)
    m = bsg.Matrix.from_system(ctx, s, symm_upper=True)
    f = bsg.Factor(ctx, m, "ich2", p)
    st = bsg.fact_stats()
    assert st["mask"] > 128 * s.n and st["members"] > 128 * s.n  # half of it on average: a triangle's rows
    ia, ja, l, uu = f.export_block()
    o = oracle.ich2_block(u.ia, u.ja, u.a, 3, tau1=3e-4, tau2=3e-4, theta=0.1)
    assert abs(p.density - o[3][0]) <= 0.01 * o[3][0]
    x = np.random.default_rng(5).standard_normal(3 * s.n)
    y, z = (oracle.solve_u_block(a, b, v, 3, oracle.solve_l_block(a, b, v, 3, x)) for a, b, v in
            ((ia, ja, uu), (o[0], o[1], o[2])))
    assert np.linalg.norm(y - z) <= 2e-2 * np.linalg.norm(z)
    f.free()
    m.free()
