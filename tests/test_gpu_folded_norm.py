"""A LayerNorm whose result only a few-row product reads is folded into that product (gemm_lanes.cu: a CTA holds whole rows; gemm_rows.cu: the
cluster puts the statistics of its parts together), and stays a launch of its own wherever something else needs its result."""
import math

import numpy as np
import pytest
import torch

from helpers import compare_outputs
from fxfusion_b200 import lowering, wire
from oracle.graph_oracle import GraphOracle

pytestmark = pytest.mark.gpu


def _run(b, tmp_path, ins):
    from fxfusion_b200.engine import ExecutionEngine
    graph = b.finish()
    path = tmp_path / "g.bin"
    wire.dump(graph, path)
    eng = ExecutionEngine(str(path), "cuda:0")
    got, want = eng.run([t.cuda() for t in ins]), GraphOracle(graph).run(ins)
    kernels = [r["kernel"] for r in eng.profile_launches()]
    assert eng.device_status() == 0
    return [g.cpu() for g in got], want, kernels, eng


# rows of one slab, a ragged last slab, parts of unequal width, the longest row; few and many columns; either kernel
@pytest.mark.parametrize("M,N,K", [(1, 512, 512), (3, 40, 64), (8, 100, 72), (32, 2304, 768), (33, 3072, 768), (17, 640, 200), (64, 1500, 1024), (5, 4096, 1000), (32, 512, 1024), (2, 7, 16)])
@pytest.mark.parametrize("op", ["Linear", "FeedForward"])
def test_folded(built_lib, tmp_path, M, N, K, op):
    rng = np.random.default_rng(M + N + K)
    b = lowering.GraphBuilder(f"norm_{M}_{N}_{K}")
    c = lambda n, k: (b.const((rng.standard_normal((n, k)) / math.sqrt(k)).astype(np.float32)), b.const(rng.standard_normal(n, dtype=np.float32)))
    x = b.input((M, K), wire.DT_F32)
    y = b.op("LayerNorm", [x, b.const(rng.standard_normal(K, dtype=np.float32)), b.const(rng.standard_normal(K, dtype=np.float32))], (M, K), ints=[1, K], floats=[1e-5])
    y = b.op("LinearRelu", [y, *c(N, K)], (M, N)) if op == "Linear" else b.op("FeedForward", [y, *c(N, K), *c(K, N)], (M, K))
    b.output(b.op("Relu", [y], (M, N if op == "Linear" else K)))
    gen = torch.Generator().manual_seed(K)
    xin = (torch.randn(M, K, generator=gen) + 2) * torch.logspace(-1, 3, M).reshape(M, 1)   # rows of very different size, away from zero
    got, want, kernels, eng = _run(b, tmp_path, [xin])
    assert "LayerNorm" not in kernels, kernels
    lines = eng.describe().splitlines()[-3:]
    assert lines[0].endswith("folded into a later node") and "+LayerNorm(node 0)" in lines[1], lines
    ok, info = compare_outputs(got[0], want[0], atol=5e-5, rtol=2e-4)
    assert ok, info
    # a row without variance is beta whatever its value; a row with a NaN or an infinity is NaN and no other is touched
    xin[0] = 0.5
    if M > 2:
        xin[1, K // 2], xin[2, 0] = float("nan"), float("inf")
    got, want = eng.run([xin.cuda()])[0].cpu(), GraphOracle(str(tmp_path / "g.bin")).run([xin])[0]
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.isnan(want).any() == (M > 2)
    # a mean off by an ulp leaves 0.5 * 2^-24 / sqrt(1e-5) = 1e-5 in every element of the constant row: at most ten times that behind the products
    ok, info = compare_outputs(got[0], want[0], atol=1.5e-4, rtol=2e-4)
    assert ok, info
    ok, info = compare_outputs(got[3:], want[3:], atol=5e-5, rtol=2e-4)
    assert ok, info
    eng.close()


@pytest.mark.parametrize("why", ["two readers", "output", "long rows", "streamed", "no product", "tail", "input overwritten"])
def test_not_folded(built_lib, tmp_path, why):
    M, K, N = 4, 1032 if why == "long rows" else 64, {"streamed": 19200, "input overwritten": 64}.get(why, 96)
    rng = np.random.default_rng(1)
    b = lowering.GraphBuilder("norm_kept")
    c = lambda n, k: (b.const((rng.standard_normal((n, k)) / math.sqrt(k)).astype(np.float32)), b.const(rng.standard_normal(n, dtype=np.float32)))
    x = b.input((1, M, K), wire.DT_F32)
    h = b.op("Relu", [x], (1, M, K)) if why == "input overwritten" else x   # (the planner gives its place to what the product writes)
    y = b.op("LayerNorm", [h, b.const(rng.standard_normal(K, dtype=np.float32)), b.const(rng.standard_normal(K, dtype=np.float32))], (1, M, K), ints=[1, K], floats=[1e-5])
    if why == "no product":
        b.output(b.op("Relu", [y], (1, M, K)))
    elif why == "tail":
        b.output(b.op("Linear", [y, *c(N, K)], (1, M, N)))
    else:
        b.output(b.op("Relu", [b.op("LinearRelu", [y, *c(N, K)], (1, M, N))], (1, M, N)))
    if why == "two readers":
        b.output(b.op("Relu", [y], (1, M, K)))
    if why == "output":
        b.output(y)
    got, want, kernels, eng = _run(b, tmp_path, [torch.randn(1, M, K, generator=torch.Generator().manual_seed(0))])
    assert "LayerNorm" in kernels, kernels
    for g, w in zip(got, want):
        ok, info = compare_outputs(g, w, atol=2e-5, rtol=1e-4)
        assert ok, info
    eng.close()


@pytest.mark.parametrize("M,N,K", [(1, 1024, 512), (8, 256, 1024), (64, 32, 1024)])
@pytest.mark.parametrize("after", ["Relu", "residual"])
@pytest.mark.parametrize("kept", [False, True])
def test_computed_gamma_and_beta(built_lib, tmp_path, M, N, K, after, kept):
    """Gamma and beta that the graph computes die at the LayerNorm, and the planner gives their place to what the product behind it writes: a folded
    LayerNorm would read them meanwhile.  Where they live on (`kept`), it is folded and reads what the launches before it wrote."""
    from fxfusion_b200.engine import ExecutionEngine
    rng = np.random.default_rng(N)
    b = lowering.GraphBuilder(f"computed_{M}_{N}_{K}")
    x, r, gin, bin_ = b.input((M, K), wire.DT_F32), b.input((M, N), wire.DT_F32), b.input((K,), wire.DT_F32), b.input((K,), wire.DT_F32)
    gamma, beta = b.op("Relu", [gin], (K,)), b.op("Relu", [bin_], (K,))
    y = b.op("LayerNorm", [x, gamma, beta], (M, K), ints=[1, K], floats=[1e-5])
    w = [b.const((rng.standard_normal((N, K)) / math.sqrt(K)).astype(np.float32)), b.const(rng.standard_normal(N, dtype=np.float32))]
    z = b.op("Linear", [y, *w], (M, N)) if after == "residual" else b.op("LinearRelu", [y, *w], (M, N))
    z2 = b.op("Add", [z, r], (M, N)) if after == "residual" else z
    b.output(b.op("Relu", [z2], (M, N)))
    if kept:
        b.output(b.op("Add", [gamma, beta], (K,)))
    graph = b.finish()
    place = lambda v: (graph.tensors[v].offset, graph.tensors[v].offset + graph.tensors[v].size_bytes)
    below = [v for v in (gamma, beta) for o in (z, z2) if place(v)[0] < place(o)[1] and place(o)[0] < place(v)[1]]
    assert bool(below) == (not kept)
    path = tmp_path / "g.bin"
    wire.dump(graph, path)
    eng = ExecutionEngine(str(path), "cuda:0")
    gen = torch.Generator().manual_seed(M)
    for _ in range(3):   # (every forward has a gamma and a beta of its own)
        ins = [torch.randn(M, K, generator=gen), torch.randn(M, N, generator=gen), torch.randn(K, generator=gen) + 1, torch.randn(K, generator=gen)]
        for got, want in zip(eng.run([t.cuda() for t in ins]), GraphOracle(graph).run(ins)):
            ok, info = compare_outputs(got.cpu(), want, atol=5e-5, rtol=2e-4)
            assert ok, info
    kernels = [q["kernel"] for q in eng.profile_launches()]
    assert ("LayerNorm" in kernels) == (not kept), kernels
    assert eng.device_status() == 0
    eng.close()
