"""Few-row products in fp32 FFMA (kernels/gemm_lanes.cu) at the edges of their tiles: rows and columns that do not fill one, a K that does not
fill the lanes or their groups, and the residual and ReLU of a folded node."""
import math

import numpy as np
import pytest
import torch

from fxfusion_b200 import lowering, wire

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 16), (1, 512, 512), (2, 33, 72), (3, 255, 136), (4, 1000, 2048), (5, 10, 520), (8, 513, 256), (9, 256, 264), (17, 100, 128), (31, 512, 504),
                                   (32, 300, 256), (1, 3072, 768), (1, 768, 3072), (2, 4001, 96), (64, 250, 256), (50, 256, 200)])
def test_against_fp64(built_lib, tmp_path, M, N, K):
    from fxfusion_b200.engine import ExecutionEngine
    rng = np.random.default_rng(M + N + K)
    w, bias = (rng.standard_normal((N, K)) / math.sqrt(K)).astype(np.float32), rng.standard_normal(N, dtype=np.float32)
    b = lowering.GraphBuilder(f"lanes_{M}_{N}_{K}")
    x, r = b.input((M, K), wire.DT_F32), b.input((M, N), wire.DT_F32)
    lin = b.op("Linear", [x, b.const(w), b.const(bias)], (M, N))
    b.output(b.op("AddRelu", [lin, r], (M, N)))
    b.output(b.op("LinearRelu", [x, b.const(w), b.const(bias)], (M, N)))
    path = tmp_path / "g.bin"
    wire.dump(b.finish(), path)
    eng = ExecutionEngine(str(path), "cuda:0")
    gen = torch.Generator().manual_seed(K)
    xin, rin = torch.randn(M, K, generator=gen), torch.randn(M, N, generator=gen)
    xin *= 10.0 ** torch.linspace(-6, 6, K)
    if M > 1:
        xin[M - 1, K // 2] = float("nan")
    got = [t.cpu().double() for t in eng.run([xin.cuda(), rin.cuda()])]
    y = xin.double() @ torch.from_numpy(w).double().T + torch.from_numpy(bias).double()
    # K / 32 additions in a lane, 13 over lanes and groups, two more for bias and residual, each within half an ulp of what it adds up
    size = xin.abs().double() @ torch.from_numpy(w).abs().double().T + torch.from_numpy(bias).abs().double()
    for g, want, top in ((got[0], torch.relu(y + rin.double()), size + rin.abs().double()), (got[1], torch.relu(y), size)):
        assert torch.equal(torch.isnan(g), torch.isnan(want))
        seen = ~torch.isnan(want)
        assert ((g - want).abs()[seen] <= ((K / 32 + 15) * 2.0 ** -24 * top)[seen]).all()
    eng.profile_launches()
    assert all(q["kernel"] == "gemm_lanes_ffma" for q in eng.profile_launches())
    assert eng.device_status() == 0
    eng.close()


# On either side of what the rule was measured for (rows, columns, K)
@pytest.mark.parametrize("M,N,K,lanes", [(1, 9472, 64, True), (1, 9473, 64, False), (1, 16000, 64, False), (8, 9000, 64, True), (8, 64, 1408, True), (8, 64, 1416, False), (4, 64, 1416, True),
                                         (9, 3072, 32, True), (9, 3073, 32, False), (9, 64, 1032, False), (32, 3000, 32, False), (64, 704, 704, False), (64, 16000, 64, False)])
def test_dispatch(built_lib, tmp_path, M, N, K, lanes):
    from fxfusion_b200.engine import ExecutionEngine
    rng = np.random.default_rng(M + N + K)
    w, bias = (rng.standard_normal((N, K)) / math.sqrt(K)).astype(np.float32), rng.standard_normal(N, dtype=np.float32)
    b = lowering.GraphBuilder(f"rule_{M}_{N}_{K}")
    x = b.input((M, K), wire.DT_F32)
    b.output(b.op("Relu", [b.op("LinearRelu", [x, b.const(w), b.const(bias)], (M, N))], (M, N)))
    path = tmp_path / "g.bin"
    wire.dump(b.finish(), path)
    eng = ExecutionEngine(str(path), "cuda:0")
    xin = torch.randn(M, K, generator=torch.Generator().manual_seed(K))
    got = eng.run([xin.cuda()])[0].cpu().double()
    want = torch.relu(xin.double() @ torch.from_numpy(w).double().T + torch.from_numpy(bias).double())
    assert ((got - want).norm() / want.norm()).item() < 2.0 ** -20   # 22 bits of each factor, at most K / 16 truncated additions
    assert [q["kernel"] for q in eng.profile_launches()][0].startswith("gemm_lanes_ffma" if lanes else "gemm_f16x3"), eng.describe()
    assert eng.device_status() == 0
    eng.close()
