"""Block products of five, six and more vectors over the lengths of the block rows:
the interleaved form (csrc/k_spmv.cu) is taken where there are blocks enough to pay
for it, or vectors beyond L2.  Every vector gets the bits of its own product, and
bsg_launch_count tells the form: the interleaved one is two launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,interleaved", [
    (6000, 1, False), (6000, 21, False), (6000, 22, True), (20000, 2, False), (20000, 9, False), (20000, 10, True),
    (60000, 4, False), (60000, 7, True), (399999, 1, False), (400000, 1, True)])
def test_form_by_row_length(ctx, n, k, interleaved):
    import bsg
    import torch
    rng = np.random.default_rng(k)
    off = np.concatenate([[0], 1 + rng.choice(3000, k - 1, replace=False)])
    ja = (np.arange(n)[:, None] + off[None, :]) % n
    ja = np.concatenate([ja[:, :1], np.sort(ja[:, 1:], axis=1)], axis=1)
    m = bsg.Matrix(ctx, n, np.arange(n + 1) * k, ja.ravel(), rng.standard_normal(9 * n * k), 3, False)
    for nr, forms in ((6, 1), (5, 1), (11, 2)):
        X = torch.randn((nr, 3 * n), generator=torch.Generator(device="cuda").manual_seed(nr), dtype=torch.float64,
                        device="cuda")
        Y, y = torch.full_like(X, float("nan")), torch.empty_like(X[0])
        before = bsg.lib().bsg_launch_count()
        m.mvm_multi(X, Y)
        assert bsg.lib().bsg_launch_count() - before == forms * (2 if interleaved else 1)
        for q in (0, nr // 2, nr - 1):
            m.mvm(X[q], y)
            assert torch.equal(y, Y[q]), q
    m.free()
