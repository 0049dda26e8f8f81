"""The tensor-core attention kernel (kernels/attention_tc.cu) at sequence lengths whose mask rows and V^T rows are not aligned:
mask bytes at any address, key blocks and query tiles with a remainder, blocks that may be skipped and blocks that may not."""
import math

import numpy as np
import pytest
import torch

from helpers import compare_outputs
from fxfusion_b200 import lowering, wire
from oracle.graph_oracle import GraphOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [17, 63, 65, 127, 129, 198, 259])
@pytest.mark.parametrize("kind", ["causal", "blocks", "keys"])
def test_any_sequence_length(built_lib, tmp_path, T, kind):
    from fxfusion_b200.engine import ExecutionEngine
    B, H, D = 3, 2, 128
    rng = np.random.default_rng(T)
    mat = lambda n, k: (rng.standard_normal((n, k)) / math.sqrt(k)).astype(np.float32)
    b = lowering.GraphBuilder(f"attn_{T}_{kind}")
    x = b.input((B, T, D), wire.DT_F32)
    m = b.input((B, 1, T, T) if kind != "keys" else (B, 1, 1, T), wire.DT_BOOL)
    b.output(b.op("MHA", [x, m, b.const(mat(3 * D, D)), b.const(rng.standard_normal(3 * D, dtype=np.float32)), b.const(mat(D, D)), b.const(rng.standard_normal(D, dtype=np.float32))],
                  (B, T, D), ints=[H, 64, D, 3 * D], floats=[8.0]))
    graph = b.finish()
    path = tmp_path / "g.bin"
    wire.dump(graph, path)
    eng = ExecutionEngine(str(path), "cuda:0")
    gen = torch.Generator().manual_seed(T)
    xin = torch.randn(B, T, D, generator=gen)
    if kind == "causal":
        mask = torch.tril(torch.ones(T, T, dtype=torch.bool)).expand(B, 1, T, T).contiguous()
    elif kind == "blocks":
        mask = torch.rand(B, 1, T, T, generator=gen) < 0.3
        mask[:, :, :, :T // 2] = False      # whole blocks of keys that no query sees
        mask[..., T - 1] = True
        mask[1, 0, T - 1] = False           # a row that sees nothing: NaN
    else:
        mask = torch.rand(B, 1, 1, T, generator=gen) < 0.7
        mask[..., 0] = True
    got, want = eng.run([xin.cuda(), mask.cuda()])[0].cpu(), GraphOracle(graph).run([xin, mask])[0]
    ok, info = compare_outputs(got, want, atol=2e-5, rtol=2e-4)
    assert ok, info
    eng.profile_launches()
    assert any("attention_tf32" in r["kernel"] for r in eng.profile_launches())
    xin[2, T // 3] = float("inf")           # reaches every row of the batch through 0 * inf, a skipped block or not
    got, want = eng.run([xin.cuda(), mask.cuda()])[0].cpu(), GraphOracle(graph).run([xin, mask])[0]
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert eng.device_status() == 0
    eng.close()


@pytest.mark.parametrize("precision", ["auto", "bf16"])
@pytest.mark.parametrize("B,T,Tk", [(2, 65, 65), (3, 40, 17), (1, 200, 130), (5, 256, 64), (3, 33, 96)])
def test_context_leaves_in_split_form(built_lib, tmp_path, B, T, Tk, precision):
    """LayerNorm -> MHA -> LayerNorm -> CrossMHA over a normalised memory: neither context passes through a conversion kernel."""
    from fxfusion_b200.engine import ExecutionEngine
    D = 128
    rng = np.random.default_rng(T)
    b = lowering.GraphBuilder(f"attn_split_{B}_{T}_{Tk}")
    c = lambda n, k: (b.const((rng.standard_normal((n, k)) / math.sqrt(k)).astype(np.float32)), b.const(rng.standard_normal(n, dtype=np.float32)))
    norm = lambda v, L: b.op("LayerNorm", [v, b.const(rng.standard_normal(D, dtype=np.float32)), b.const(rng.standard_normal(D, dtype=np.float32))], (B, L, D), ints=[1, D], floats=[1e-5])
    x, mem = b.input((B, T, D), wire.DT_F32), b.input((B, Tk, D), wire.DT_F32)
    m, mk = b.input((B, 1, 1, T), wire.DT_BOOL), b.input((B, 1, 1, Tk), wire.DT_BOOL)
    h = b.op("MHA", [norm(x, T), m, *c(3 * D, D), *c(D, D)], (B, T, D), ints=[2, 64, D, 3 * D], floats=[8.0])
    b.output(b.op("CrossMHA", [norm(h, T), norm(mem, Tk), mk, *c(D, D), *c(2 * D, D), *c(D, D)], (B, T, D), ints=[2, 64, D, 2 * D], floats=[8.0]))
    graph = b.finish()
    path = tmp_path / "g.bin"
    wire.dump(graph, path)
    eng = ExecutionEngine(str(path), "cuda:0", precision=precision)
    gen = torch.Generator().manual_seed(T)
    ins = [torch.randn(B, T, D, generator=gen), torch.randn(B, Tk, D, generator=gen) * 1e3, torch.rand(B, 1, 1, T, generator=gen) < 0.8, torch.rand(B, 1, 1, Tk, generator=gen) < 0.8]
    ins[2][..., 0] = ins[3][..., 0] = True
    ins[3][B - 1] = False                   # a batch that sees nothing: NaN
    got, want = eng.run([t.cuda() for t in ins])[0].cpu(), GraphOracle(graph).run(ins)[0]
    if precision == "auto":
        ok, info = compare_outputs(got, want, atol=5e-5, rtol=2e-4)
        assert ok, info
    else:
        assert torch.equal(torch.isnan(got), torch.isnan(want))
        assert ((got - want)[:B - 1].abs().max() / want[:B - 1].abs().max()).item() < 3e-2 if B > 1 else True
    eng.profile_launches()
    kernels = [r["kernel"] for r in eng.profile_launches()]
    assert not any("split_rows" in k for k in kernels) or B * T <= 64 or B * Tk <= 64, kernels
    assert eng.device_status() == 0
    eng.close()
