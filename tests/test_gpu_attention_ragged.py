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
