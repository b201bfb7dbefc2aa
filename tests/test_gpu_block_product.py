"""Block products of several vectors (csrc/k_spmv.cu): the interleaved form that
five and six vectors of larger systems take, at and around the row count and the
vector counts where it changes over, against the single-vector product (the same
bits) and in a captured graph, where it is not taken."""
import pytest

import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nn", [4, 18, 19])  # 64, 5832 and 6859 block rows
@pytest.mark.parametrize("nr", [4, 5, 6, 7, 8, 9, 11, 13, 14])
def test_vectors_equal_single_products(ctx, nn, nr):
    import bsg
    import torch
    s = P.lame3d(nn, sigma=0.5, seed=2)
    m = bsg.Matrix(ctx, s.n, s.ia, s.ja, s.a, 3, False)
    g = torch.Generator(device="cuda").manual_seed(nr)
    X = torch.randn((nr, 3 * s.n), generator=g, dtype=torch.float64, device="cuda")
    Y, y = torch.full_like(X, float("nan")), torch.empty_like(X[0])
    m.mvm_multi(X, Y)
    for q in range(nr):
        m.mvm(X[q].contiguous(), y)
        assert torch.equal(y, Y[q]), q
    m.free()


def test_vectors_in_a_captured_graph():
    import bsg
    import torch
    s = P.lame3d(20, sigma=0.5, seed=2)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        c = bsg.Context(0, st.cuda_stream)
        m = bsg.Matrix(c, s.n, s.ia, s.ja, s.a, 3, False)
        X = torch.randn((6, 3 * s.n), dtype=torch.float64, device="cuda")
        Y, Z = torch.empty_like(X), torch.empty_like(X)
        m.mvm_multi(X, Y)
        st.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            m.mvm_multi(X, Z)
        X.normal_()
        m.mvm_multi(X, Y)
        graph.replay()
        st.synchronize()
        assert torch.equal(Y, Z)
        del graph
        m.free()
        c.close()
