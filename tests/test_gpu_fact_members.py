"""Point factorisation (csrc/k_fact.cu): members taken one by one as they
finish, and the columns kept in order while a row waits.  Factors are compared
bit for bit with the oracle where those paths change over: rows of more than 32
and of more than 64 stored entries (lower thresholds), members farther than the
16384 rows of the member bitmap, rows of one and two entries, a chain, and rows
whose dropped columns are 0 .. 8 modulo the groups of 8 they are added in."""
import numpy as np
import pytest

import problems as P

pytestmark = pytest.mark.gpu

CASES = {
    "chain": (P.heat3d, (400, 1, 1), 0.7, 1e-3, 1e-3),
    "pair": (P.heat3d, (2, 1, 1), 0.5, 1e-3, 1e-3),
    "rows of 30": (P.heat3d, (11, 10, 9), 1.0, 1e-3, 1e-3),
    "rows of 60": (P.heat3d, (11, 10, 9), 0.5, 2e-4, 2e-4),
    "rows of 100": (P.heat3d, (9, 9, 9), 0.3, 2e-5, 2e-5),
    "second order": (P.heat3d, (9, 8, 7), 1.0, 1e-2, 1e-4),
    "few kept": (P.heat3d, (10, 9, 8), 1.0, 2e-1, 1e-3),
    "far members": (P.heat3d, (17000, 3, 1), 1.0, 1e-3, 1e-3),
    "wide 2-D": (P.heat3d, (130, 70, 1), 1.2, 1e-3, 1e-3),
}


@pytest.mark.parametrize("kind", ["ich2", "ilu2"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_factor_equals_oracle(ctx, oracle, name, kind):
    import bsg
    gen, dims, sigma, tau1, tau2 = CASES[name]
    s = gen(*dims, sigma=sigma, seed=len(name))
    u = s.upper()
    p = bsg.default_param(ordtype=0, fcttyp=2, tau1=tau1, tau2=tau2, memory=100.0)
    m = bsg.Matrix.from_system(ctx, s, symm_upper=True)
    f = bsg.Factor(ctx, m, kind, p)
    giu, gju, gl, gu = f.export()
    iu, ju, lv, uv, _ = oracle.fact(0 if kind == "ich2" else 1, u.ia, u.ja, u.a, tau1=tau1, tau2=tau2)
    assert np.array_equal(giu, iu) and np.array_equal(gju, ju)
    assert np.array_equal(gl, lv) and np.array_equal(gu, uv)
    f.free()
    m.free()
