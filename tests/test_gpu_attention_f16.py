"""Attention on Q, K and V in split form (kernels/attention_f16.cu): LayerNorm -> MHA / CrossMHA, at the edges of its tiles (128 queries, key
blocks of 64 and 128, 32 rows per finite flag), for every mask layout, with blocks that are skipped and values that are not finite."""
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


def _graph(B, T, Tk, mask, seed, gain=1.0):
    D, H = 128, 2
    rng = np.random.default_rng(seed)
    b = lowering.GraphBuilder(f"attn_f16_{T}_{Tk}")
    c = lambda n, k, s=1.0: (b.const((s * rng.standard_normal((n, k)) / math.sqrt(k)).astype(np.float32)), b.const((0.1 * rng.standard_normal(n)).astype(np.float32)))
    norm = lambda v, L: b.op("LayerNorm", [v, b.const(rng.standard_normal(D, dtype=np.float32)), b.const(rng.standard_normal(D, dtype=np.float32))], (B, L, D), ints=[1, D], floats=[1e-5])
    x = b.input((B, T, D), wire.DT_F32)
    if Tk == T:
        m = b.input(tuple(mask.shape), wire.DT_BOOL)
        b.output(b.op("MHA", [norm(x, T), m, *c(3 * D, D, gain), *c(D, D)], (B, T, D), ints=[H, 64, D, 3 * D], floats=[7.0]))
    else:
        mem = b.input((B, Tk, D), wire.DT_F32)
        m = b.input(tuple(mask.shape), wire.DT_BOOL)
        b.output(b.op("CrossMHA", [norm(x, T), norm(mem, Tk), m, *c(D, D, gain), *c(2 * D, D, gain), *c(D, D)], (B, T, D), ints=[H, 64, D, 2 * D], floats=[7.0]))
    return b.finish()


# Scores reach about 20 here; fp32 itself (the oracle) is then 1e-5 off in the exponent, which the tolerance covers.
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
@pytest.mark.parametrize("what,r", [(w, r) for w in ("thirds", "heads", "columns") for r in (1.0, 16.0, 1024.0, 3e5)] + [("thirds", 1e21)])
def test_uneven_sizes(built_lib, tmp_path, what, r, cross):
    """Q's weights divided and K's multiplied by the same factors, which leaves the function as it is: all of them by r, or by r in one head and 1 / r
    in the next, or every column by a factor of its own up to r.  Against fp64: Q, K and V keep 22 bits of what they add to a score, sum |q_d k_d| / 8
    is about 5 here, so a score is off by 5 * 2^-21 at most and a probability by that much of itself; 2^-18 covers it and the sums in fp32."""
    from fxfusion_b200.engine import ExecutionEngine
    B, T, Tk, D, H = 1, 130, 200, 384, 6
    rng = np.random.default_rng(11)
    f = {"thirds": np.full(D, r), "heads": np.repeat(r ** np.where(np.arange(H) % 2, -1.0, 1.0), 64), "columns": r ** rng.uniform(-1, 1, D)}[what].astype(np.float32)
    wq, wk, wv, wo = (rng.standard_normal((D, D)) / math.sqrt(D) for _ in range(4))
    bq, bk, bv, bo = (0.1 * rng.standard_normal(D) for _ in range(4))
    wq, bq, wk, bk = wq / f[:, None], bq / f, wk * f[:, None], bk * f
    w = [t.astype(np.float32) for t in (wq, wk, wv, wo)]
    bias = [t.astype(np.float32) for t in (bq, bk, bv, bo)]
    b = lowering.GraphBuilder(f"uneven_{what}_{r}")
    one, zero = b.const(np.ones(D, np.float32)), b.const(np.zeros(D, np.float32))
    norm = lambda v, L: b.op("LayerNorm", [v, one, zero], (B, L, D), ints=[1, D], floats=[1e-5])
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
    ln = lambda t: torch.nn.functional.layer_norm(t.double(), (D,), eps=1e-5)
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
