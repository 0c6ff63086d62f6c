"""Kernels started while the one in front of them drains: the same bits on the legacy stream, on a
stream of its own, beside another stream's products, and (FP64) replayed from a captured graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
cs = pytest.importorskip("cosmicscanner_b200")
synth = pytest.importorskip("cosmicscanner_b200.synth")


def make(n, m, k, seed):
    d = synth.cohort(n, m, seed, missing=0.02, n_causal=5, maf_lo=0.05)
    g = cs.Genotypes.from_bed_bytes(d["bed"], n, m)
    op = cs.createKinshipOperator(g)
    X = torch.from_numpy(np.random.default_rng(seed).standard_normal((k, n))).cuda()
    return g, op, X


def apply(op, X, Y, precision):
    n, k = X.shape[1], X.shape[0]
    op.apply_device(X.data_ptr(), n, k, Y.data_ptr(), n, precision, torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,m,k", [(500, 3000, 1), (700, 900, 20), (3000, 2000, 40), (600, 700, 130)])
def test_streams_and_graphs(precision, n, m, k):
    g, op, X = make(n, m, k, n)
    want = torch.empty_like(X)
    apply(op, X, want, precision)
    torch.cuda.synchronize()
    # repeated products whose input is the last one's output: each must wait for all of it
    chain = X.clone()
    for _ in range(20):
        apply(op, chain, chain, precision)
    torch.cuda.synchronize()
    again = X.clone()
    for _ in range(20):
        apply(op, again, again, precision)
        torch.cuda.synchronize()
    assert torch.equal(chain, again)
    # another operator's products on a stream of their own at the same time
    g2, op2, X2 = make(n + 3, m, k, n + 1)
    want2 = torch.empty_like(X2)
    apply(op2, X2, want2, precision)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    Y, Y2 = torch.empty_like(X), torch.empty_like(X2)
    for _ in range(10):
        apply(op, X, Y, precision)
        with torch.cuda.stream(s):
            apply(op2, X2, Y2, precision)
    torch.cuda.synchronize()
    assert torch.equal(Y, want) and torch.equal(Y2, want2)
    if precision == "mixed":
        return  # reads its status back on each call: not capturable
    graph = torch.cuda.CUDAGraph()
    out = torch.zeros_like(X)
    with torch.cuda.graph(graph):
        apply(op, X, out, precision)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
