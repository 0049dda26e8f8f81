"""Products and convolutions of one round whose tiles are cut along K inside clusters (kernels/gemm_f16.cu): tiles of every width, 2 to 8 parts of even
and uneven depth, tiles that end inside a warp's block, several chains per part, and what the finishing warps do (residual, ReLU, split form,
image maxima)."""
import math

import numpy as np
import pytest
import torch

from fxfusion_b200 import lowering, wire
from oracle.graph_oracle import GraphOracle

pytestmark = pytest.mark.gpu


def _engine(b, tmp_path, **kw):
    from fxfusion_b200.engine import ExecutionEngine
    graph = b.finish()
    path = tmp_path / "g.bin"
    wire.dump(graph, path)
    return graph, ExecutionEngine(str(path), "cuda:0", **kw)


# The cut products of each: columns of a tile, parts.  The first product of the pair leaves in split form, the second with the residual.
@pytest.mark.parametrize("M,N,K,cut", [
    (65, 32, 128, []), (70, 40, 200, []), (300, 768, 3072, []), (1000, 96, 2048, []),
    (66, 1232, 848, ["32_cut4", "32_cut2"]), (68, 368, 552, ["32_cut3"]), (129, 256, 1024, ["32_cut4"]), (512, 256, 1024, ["32_cut4"]), (100, 1000, 520, ["32_cut4"]), (150, 250, 1160, ["32_cut5"]),
    (110, 16, 368, ["32_cut6"]), (85, 40, 416, ["32_cut7"]), (128, 16, 456, ["32_cut8"]), (500, 64, 8192, ["32_cut8"]),
    (67, 1128, 1392, ["32_cut3", "64_cut6"]), (151, 808, 1336, ["64_cut3"]), (129, 552, 984, ["64_cut4"]), (67, 1160, 1208, ["64_cut5", "64_cut5"]), (333, 168, 1304, ["64_cut7"]),
    (100, 768, 3072, ["64_cut8"]), (130, 1936, 264, ["64_cut8"]),
    (134, 1216, 1600, ["128_cut5"]), (132, 1016, 1824, ["128_cut6"]), (142, 840, 1312, ["128_cut7"]), (135, 624, 1992, ["128_cut8"]), (200, 768, 3072, ["128_cut8"]),
    (137, 1992, 624, ["128_cut8"]), (200, 3072, 768, ["128_cut8"])])
def test_rows(built_lib, tmp_path, M, N, K, cut):
    """FeedForward (its hidden activation in split form) and a residual, against fp64: each of the K / 16 x 3 additions of a part truncates by up to an
    ulp of a running sum, and the parts and the rest are added in fp32."""
    rng = np.random.default_rng(M + N + K)
    w1, w2 = (rng.standard_normal((K, N)) / math.sqrt(N)).astype(np.float32), (rng.standard_normal((N, K)) / math.sqrt(K)).astype(np.float32)
    b1, b2 = rng.standard_normal(K, dtype=np.float32), rng.standard_normal(N, dtype=np.float32)
    b = lowering.GraphBuilder(f"cut_{M}_{N}_{K}")
    x = b.input((M, N), wire.DT_F32)
    ff = b.op("FeedForward", [x, *(b.const(t) for t in (w1, b1, w2, b2))], (M, N))
    b.output(b.op("AddRelu", [ff, x], (M, N)))
    graph, eng = _engine(b, tmp_path)
    assert [r["kernel"].removeprefix("gemm_f16x3_tcgen05_") for r in eng.profile_launches() if "_cut" in r["kernel"]] == cut
    xin = torch.randn(M, N, generator=torch.Generator().manual_seed(K))
    xin[M - 1, 0] = float("nan")
    d = lambda t: torch.from_numpy(t).double()
    want = torch.relu(torch.relu(xin.double() @ d(w1).T + d(b1)) @ d(w2).T + d(b2) + xin.double())
    first = eng.run([xin.cuda()])[0].cpu()
    assert torch.isnan(first[M - 1]).all() and not torch.isnan(first[:M - 1]).any()
    got = first[:M - 1].double()
    assert ((got - want[:M - 1]).norm() / want[:M - 1].norm()).item() < 2.0 ** -19
    for _ in range(3):   # parts are added in a fixed order
        assert torch.equal(eng.run([xin.cuda()])[0].cpu()[:M - 1], first[:M - 1])
    assert eng.device_status() == 0
    eng.close()


# Of the three convolutions behind the stem (1x1, k x k with the residual, 1x1 into fp32 pixels) those that are cut: columns of a tile, parts.
@pytest.mark.parametrize("N,size,C,O,k,s,cut", [
    (4, 17, 1024, 136, 1, 1, ["32_cut2", "32_cut2"]), (3, 5, 64, 512, 3, 1, ["32_cut3", "32_cut8"]), (3, 13, 64, 64, 3, 1, ["32_cut5"]),
    (3, 5, 128, 32, 3, 1, ["32_cut6"]), (4, 5, 64, 40, 5, 1, ["32_cut7"]), (2, 14, 512, 136, 3, 2, ["32_cut8", "32_cut8"]),
    (2, 7, 1024, 256, 1, 1, ["32_cut8", "32_cut8"]), (1, 28, 128, 256, 3, 1, ["64_cut3"]), (1, 28, 256, 256, 3, 1, ["64_cut4"]),
    (2, 12, 128, 512, 3, 1, ["64_cut5", "32_cut8"]), (1, 14, 512, 512, 3, 1, ["64_cut6", "32_cut8"]), (1, 23, 2048, 1024, 1, 1, ["128_cut3", "128_cut3", "32_cut8"]),
    (4, 14, 512, 512, 3, 1, ["128_cut4", "32_cut4"]), (2, 12, 512, 1024, 3, 1, ["128_cut5", "32_cut8"]), (4, 14, 512, 256, 3, 1, ["128_cut8"])])
def test_images(built_lib, tmp_path, N, size, C, O, k, s, cut):
    rng = np.random.default_rng(size + C)
    gb = [1, 1, 1, 256, 1, 1]
    b = lowering.GraphBuilder(f"cut_images_{N}_{size}_{C}_{O}")

    def conv(x, c, o, h, kk, ss, pad):
        ho = (h + 2 * pad - kk) // ss + 1
        w = (rng.standard_normal((o, c, kk, kk)) / math.sqrt(c * kk * kk)).astype(np.float32)
        return b.op("Conv2d", [x, b.const(w), b.const(rng.standard_normal(o, dtype=np.float32))], (N, o, ho, ho), ints=[ss, ss, pad, pad, 1, 1, 1] + gb), ho

    x = b.input((N, 3, size * 2, size * 2), wire.DT_F32)
    y, h = conv(x, 3, C, size * 2, 7, 2, 3)
    r, _ = conv(y, C, O, h, 1, s, 0)
    z, h2 = conv(y, C, O, h, k, s, k // 2)
    z = b.op("AddRelu", [z, r], (N, O, h2, h2))
    p = b.op("AvgPool2d", [conv(z, O, 24, h2, 1, 1, 0)[0]], (N, 24, h2, h2), ints=[1, 1, 1, 1, 0, 0, 0] + gb)   # (reads fp32 pixels)
    b.output(conv(p, 24, 8, h2, 1, 1, 0)[0])
    b.output(b.op("AdaptiveAvgPool2d", [z], (N, O, 1, 1), ints=[1, 1] + gb))
    b.output(b.op("AdaptiveAvgPool2d", [y], (N, C, 1, 1), ints=[1, 1] + gb))   # y lives on: in its place the sum could not join the convolution
    graph, eng = _engine(b, tmp_path)
    text = eng.describe()
    assert text.count("output in split form") == 3 and "+AddRelu(residual" in text, text
    assert [q["kernel"].removeprefix("conv2d_f16x3_tcgen05_") for q in eng.profile_launches() if "_cut" in q["kernel"] and q["node"] > 0] == cut
    xin = torch.randn(N, 3, size * 2, size * 2, generator=torch.Generator().manual_seed(3)) * 10.0 ** torch.linspace(-3, 3, N).reshape(N, 1, 1, 1)
    got, want = eng.run([xin.cuda()]), GraphOracle(graph).run([xin])
    for g, t in zip(got, want):
        assert ((g.cpu() - t).abs() / t.abs().amax(dim=(1, 2, 3), keepdim=True)).max().item() < 6e-6
    first = [g.cpu() for g in got]
    for _ in range(3):
        assert all(torch.equal(a.cpu(), f) for a, f in zip(eng.run([xin.cuda()]), first))
    assert eng.device_status() == 0
    eng.close()
