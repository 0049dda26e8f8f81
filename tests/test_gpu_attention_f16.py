"""Attention on Q, K and V in split form (kernels/attention_f16.cu): LayerNorm -> MHA / CrossMHA, at the edges of its tiles (128 queries, key
blocks of 64 and 128, each with a finite flag per batch; the most keys), for every mask layout, with blocks that are skipped and values that are not
finite; and what still runs on the kernel for fp32 rows (kernels/attention_tc.cu)."""
import math

import numpy as np
import pytest
import torch

from helpers import compare_outputs
from fxfusion_b200 import lowering, wire
from oracle.graph_oracle import GraphOracle

pytestmark = pytest.mark.gpu


def _mask(kind, B, H, T, Tk, gen):
    if kind == "causal":
        return torch.tril(torch.ones(T, Tk, dtype=torch.bool)).expand(B, 1, T, Tk).contiguous()
    if kind == "keys":
        m = torch.rand(B, 1, 1, Tk, generator=gen) < 0.7
        m[..., 0] = True
    elif kind == "queries":                 # one byte for all keys of a query: rows see everything or nothing
        m = torch.rand(1, H, T, 1, generator=gen) < 0.8
    else:                                   # per head, the first half of the keys unseen by all, one batch that sees nothing
        m = torch.rand(B, H, T, Tk, generator=gen) < 0.3
        m[..., :Tk // 2] = False
        m[..., Tk - 1] = True
        m[B - 1] = False
    return m


def _graph(B, T, Tk, mask, seed):
    D, H = 128, 2
    rng = np.random.default_rng(seed)
    b = lowering.GraphBuilder(f"attn_f16_{T}_{Tk}")
    c = lambda n, k: (b.const((rng.standard_normal((n, k)) / math.sqrt(k)).astype(np.float32)), b.const((0.1 * rng.standard_normal(n)).astype(np.float32)))
    norm = lambda v, L: b.op("LayerNorm", [v, b.const(rng.standard_normal(D, dtype=np.float32)), b.const(rng.standard_normal(D, dtype=np.float32))], (B, L, D), ints=[1, D], floats=[1e-5])
    x = b.input((B, T, D), wire.DT_F32)
    if Tk == T:
        m = b.input(tuple(mask.shape), wire.DT_BOOL)
        b.output(b.op("MHA", [norm(x, T), m, *c(3 * D, D), *c(D, D)], (B, T, D), ints=[H, 64, D, 3 * D], floats=[7.0]))
    else:
        mem = b.input((B, Tk, D), wire.DT_F32)
        m = b.input(tuple(mask.shape), wire.DT_BOOL)
        b.output(b.op("CrossMHA", [norm(x, T), norm(mem, Tk), m, *c(D, D), *c(2 * D, D), *c(D, D)], (B, T, D), ints=[H, 64, D, 2 * D], floats=[7.0]))
    return b.finish()


def _f64(graph, ins):
    """The oracle's kernels in 64 bits."""
    o = GraphOracle(graph)
    o.reg = [t.double() if t is not None and t.dtype == torch.float32 else t for t in o.reg]
    for t in graph.tensors:
        if t.kind in (wire.KIND_ALIAS, wire.KIND_OUTPUT) and t.alias_of >= 0:
            o.reg[t.id] = o.reg[t.alias_of].view(list(t.shape))
    return o.run(ins)[0]


# Element by element against the oracle: scores reach about 20 here, fp32 itself is then 1e-5 off in the exponent, which the tolerance covers.
# As a whole against fp64: Q, K and V keep 22 bits of what they add to a score; sum |q_d k_d| / 7 is 10 to 20 where gamma is N(0, 1), so a
# probability is off by 20 * 2^-21 of itself at most, the context and the output by that much of theirs.
@pytest.mark.parametrize("precision", ["auto", "bf16"])
@pytest.mark.parametrize("kind", ["causal", "keys", "queries", "blocks"])
@pytest.mark.parametrize("B,T,Tk", [(5, 16, 16), (3, 63, 63), (2, 64, 64), (3, 65, 65), (2, 127, 127), (2, 128, 128), (3, 129, 129), (2, 198, 198), (1, 256, 256), (2, 300, 300),
                                    (1, 1024, 1024), (9, 8, 130), (3, 130, 22), (2, 257, 513)])
def test_matches_oracle(built_lib, tmp_path, B, T, Tk, kind, precision):
    from fxfusion_b200.engine import ExecutionEngine
    gen = torch.Generator().manual_seed(T * 7 + Tk)
    mask = _mask(kind, B, 2, T, Tk, gen)
    graph = _graph(B, T, Tk, mask, T + Tk)
    path = tmp_path / "g.bin"
    wire.dump(graph, path)
    eng = ExecutionEngine(str(path), "cuda:0", precision=precision)
    ins = [torch.randn(B, T, 128, generator=gen)] + ([] if Tk == T else [torch.randn(B, Tk, 128, generator=gen) * 1e3]) + [mask]
    for _ in range(2):
        got, want = eng.run([t.cuda() for t in ins])[0].cpu(), GraphOracle(graph).run(ins)[0]
        assert torch.equal(torch.isnan(got), torch.isnan(want))
        if precision == "auto":
            ok, info = compare_outputs(got, want, atol=5e-5, rtol=2e-4)
            assert ok, info
            seen, exact = ~torch.isnan(want), _f64(graph, ins)
            assert not seen.any() or ((got - exact)[seen].norm() / exact[seen].norm()).item() < 20 * 2.0 ** -21
        else:                               # 8 bits in the projections
            seen = ~torch.isnan(want)
            assert not seen.any() or ((got - want)[seen].norm() / want[seen].norm()).item() < 2e-2
        ins[-2] = ins[-2].clone()
        ins[-2][0, (Tk if Tk != T else T) // 3] = float("inf")   # reaches every row of its batch, a skipped block or not
    eng.profile_launches()
    assert any("attention_f16x3" in r["kernel"] for r in eng.profile_launches())
    assert eng.device_status() == 0
    eng.close()


def test_masked_keys_do_not_move_a_bit(built_lib, tmp_path):
    """What a query does not see must not change its result: neither through a scale nor through a skipped block."""
    from fxfusion_b200.engine import ExecutionEngine
    B, T = 2, 160
    gen = torch.Generator().manual_seed(1)
    mask = torch.tril(torch.ones(T, T, dtype=torch.bool)).expand(B, 1, T, T).contiguous()
    graph = _graph(B, T, T, mask, 3)
    path = tmp_path / "g.bin"
    wire.dump(graph, path)
    eng = ExecutionEngine(str(path), "cuda:0")
    x = torch.randn(B, T, 128, generator=gen)
    a = eng.run([x.cuda(), mask.cuda()])[0].cpu()
    x[:, 100:] = torch.randn(B, 60, 128, generator=gen) * 50
    b = eng.run([x.cuda(), mask.cuda()])[0].cpu()
    assert torch.equal(a[:, :100], b[:, :100]) and not torch.equal(a[:, 100:], b[:, 100:])
    eng.close()


@pytest.mark.parametrize("cross", [False, True])
@pytest.mark.parametrize("what,r", [(w, r) for w in ("thirds", "heads", "columns") for r in (1.0, 16.0, 1024.0, 3e5)] + [("gamma", 64.0), ("thirds", 1e21)])
def test_uneven_sizes(built_lib, tmp_path, what, r, cross):
    """Q's weights divided and K's multiplied by the same factors, which leaves the function as it is: all of them by r, or by r in one head and 1 / r
    in the next, or every column by a factor of its own up to r; or gamma's entries against the weights' columns.  Against fp64: Q, K and V keep 22 bits of what they add to a score, sum |q_d k_d| / 8
    is about 5 here, so a score is off by 5 * 2^-21 at most and a probability by that much of itself; 2^-18 covers it and the sums in fp32."""
    from fxfusion_b200.engine import ExecutionEngine
    B, T, Tk, D, H = 1, 130, 200, 384, 6
    rng = np.random.default_rng(11)
    f = {"thirds": np.full(D, r), "heads": np.repeat(r ** np.where(np.arange(H) % 2, -1.0, 1.0), 64), "columns": r ** rng.uniform(-1, 1, D), "gamma": np.ones(D)}[what].astype(np.float32)
    g = (r ** rng.uniform(-1, 1, D) if what == "gamma" else np.ones(D)).astype(np.float32)
    wq, wk, wv, wo = (rng.standard_normal((D, D)) / math.sqrt(D) for _ in range(4))
    bq, bk, bv, bo = (0.1 * rng.standard_normal(D) for _ in range(4))
    wq, bq, wk, bk, wv = wq / f[:, None] / g, bq / f, wk * f[:, None] / g, bk * f, wv / g
    w = [t.astype(np.float32) for t in (wq, wk, wv, wo)]
    bias = [t.astype(np.float32) for t in (bq, bk, bv, bo)]
    b = lowering.GraphBuilder(f"uneven_{what}_{r}")
    gamma, zero = b.const(g), b.const(np.zeros(D, np.float32))
    norm = lambda v, L: b.op("LayerNorm", [v, gamma, zero], (B, L, D), ints=[1, D], floats=[1e-5])
    x = b.input((B, T, D), wire.DT_F32)
    if cross:
        mem = b.input((B, Tk, D), wire.DT_F32)
        m = b.input((1, 1, T, Tk), wire.DT_BOOL)
        b.output(b.op("CrossMHA", [norm(x, T), norm(mem, Tk), m, b.const(w[0]), b.const(bias[0]), b.const(np.concatenate(w[1:3])), b.const(np.concatenate(bias[1:3])), b.const(w[3]),
                                   b.const(bias[3])], (B, T, D), ints=[H, 64, D, 2 * D], floats=[8.0]))
    else:
        Tk = T
        m = b.input((1, 1, T, T), wire.DT_BOOL)
        b.output(b.op("MHA", [norm(x, T), m, b.const(np.concatenate(w[:3])), b.const(np.concatenate(bias[:3])), b.const(w[3]), b.const(bias[3])], (B, T, D), ints=[H, 64, D, 3 * D], floats=[8.0]))
    path = tmp_path / "g.bin"
    wire.dump(b.finish(), path)
    eng = ExecutionEngine(str(path), "cuda:0")
    gen = torch.Generator().manual_seed(5)
    xin, min_ = torch.randn(B, T, D, generator=gen), torch.randn(B, Tk, D, generator=gen)
    mask = torch.ones(1, 1, T, Tk, dtype=torch.bool).tril(Tk - T)
    got = eng.run([xin.cuda(), min_.cuda(), mask.cuda()] if cross else [xin.cuda(), mask.cuda()])[0].cpu().double()
    ln = lambda t: torch.nn.functional.layer_norm(t.double(), (D,), eps=1e-5) * torch.from_numpy(g).double()
    rows = ln(min_) if cross else ln(xin)
    d = lambda a: torch.from_numpy(a).double()
    heads = lambda t, i: (t @ d(w[i]).T + d(bias[i])).view(B, -1, H, 64).transpose(1, 2)
    s = (heads(ln(xin), 0) @ heads(rows, 1).transpose(-1, -2) / 8.0).masked_fill(~mask, float("-inf"))
    want = (torch.softmax(s, -1) @ heads(rows, 2)).transpose(1, 2).reshape(B, T, D) @ d(w[3]).T + d(bias[3])
    # (what scales of fp16 pairs cannot serve runs on the kernel for fp32 rows, whose 19 bits count here as 22 do above: 2^-15)
    beyond = r > 1e20
    assert ((got - want).norm() / want.norm()).item() < 2.0 ** (-15 if beyond else -18)
    assert ("on Q, K and V in split form" in eng.describe()) != beyond, eng.describe()
    kernels = [q["kernel"] for q in eng.profile_launches()]
    assert any(("attention_tf32" if beyond else "attention_f16x3") in k for k in kernels), kernels
    assert eng.device_status() == 0
    eng.close()


def _attention(tmp_path, q_norm, kv_norm, B, T, Tk, D, H):
    """MHA (Tk == 0) or CrossMHA whose rows come from a LayerNorm or, split by a pass of their own, from an input; in the default arithmetic."""
    from fxfusion_b200.engine import ExecutionEngine
    rng = np.random.default_rng(T + Tk + D)
    b = lowering.GraphBuilder(f"attn_{q_norm}_{kv_norm}_{T}_{Tk}_{D}")
    c = lambda n, k: (b.const((rng.standard_normal((n, k)) / math.sqrt(k)).astype(np.float32)), b.const((0.1 * rng.standard_normal(n)).astype(np.float32)))
    rows = lambda v, L, norm: b.op("LayerNorm", [v, b.const(rng.standard_normal(D, dtype=np.float32)), b.const(rng.standard_normal(D, dtype=np.float32))], (B, L, D), ints=[1, D], floats=[1e-5]) if norm else v
    gen = torch.Generator().manual_seed(T)
    ins = [torch.randn(B, L, D, generator=gen) for L in ((T, Tk) if Tk else (T,))] + [torch.ones(1, 1, T, Tk or T, dtype=torch.bool).tril((Tk or T) - T)]
    x = [b.input(tuple(t.shape), wire.DT_F32) for t in ins[:-1]]
    m = b.input(tuple(ins[-1].shape), wire.DT_BOOL)
    if Tk:
        b.output(b.op("CrossMHA", [rows(x[0], T, q_norm), rows(x[1], Tk, kv_norm), m, *c(D, D), *c(2 * D, D), *c(D, D)], (B, T, D), ints=[H, 64, D, 2 * D], floats=[8.0]))
    else:
        b.output(b.op("MHA", [rows(x[0], T, q_norm), m, *c(3 * D, D), *c(D, D)], (B, T, D), ints=[H, 64, D, 3 * D], floats=[8.0]))
    graph = b.finish()
    path = tmp_path / "g.bin"
    wire.dump(graph, path)
    eng = ExecutionEngine(str(path), "cuda:0")
    got, want = eng.run([t.cuda() for t in ins])[0].cpu().double(), _f64(graph, ins)
    kernels = [q["kernel"] for q in eng.profile_launches()]
    assert eng.device_status() == 0
    eng.close()
    return ((got - want).norm() / want.norm()).item(), kernels


# Up to 2048 keys; the last block whole, short of a key, and one key into the next.  (The bound: see test_matches_oracle; 2^-15: see test_uneven_sizes.)
@pytest.mark.parametrize("Tk,kernel,bound", [(2047, "attention_f16x3", 20 * 2.0 ** -21), (2048, "attention_f16x3", 20 * 2.0 ** -21), (2049, "attention_tf32", 2.0 ** -15)])
@pytest.mark.parametrize("cross", [False, True])
def test_most_keys(built_lib, tmp_path, Tk, kernel, bound, cross):
    off, kernels = _attention(tmp_path, True, True, 1, 130 if cross else Tk, Tk if cross else 0, 128, 2)
    assert any(kernel in k for k in kernels) and not any("split_rows" in k for k in kernels), kernels
    assert off < bound


@pytest.mark.parametrize("T,transposed", [(128, True), (100, False)])
def test_rows_that_no_layer_norm_bounds(built_lib, tmp_path, T, transposed):
    """The product on split operands writes V transposed for the kernel for fp32 rows where the sequence length is a multiple of 32; its context is split
    by a pass of its own."""
    off, kernels = _attention(tmp_path, False, False, 4, T, 0, 768, 12)
    assert any("attention_tf32" in k for k in kernels) and any("gemm_f16x3" in k for k in kernels), kernels
    assert ("attention_v_transpose" not in kernels) == transposed and kernels.count("split_rows_f16") == 2, kernels
    assert off < 2.0 ** -15


@pytest.mark.parametrize("T,Tk", [(130, 200), (128, 128 * 3)])
def test_only_the_keys_are_bounded(built_lib, tmp_path, T, Tk):
    """Queries as they come, keys and values behind a LayerNorm: the kernel for fp32 rows, whose context leaves in split form under V's bound."""
    off, kernels = _attention(tmp_path, False, True, 2, T, Tk, 384, 6)
    assert any("attention_tf32" in k for k in kernels) and kernels.count("split_rows_f16") == 1, kernels
    assert off < 2.0 ** -15
