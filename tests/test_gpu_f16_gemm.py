"""The f16 GEMM (kernels/gemm_f16.cu) and the split form of its operands: every tile variant at its edges, rows of any scale,
and activations that stay in split form between the nodes of an engine."""
import math

import numpy as np
import pytest
import torch

from helpers import compare_outputs
from fxfusion_b200 import lowering, wire
from oracle.graph_oracle import GraphOracle

pytestmark = pytest.mark.gpu
ATOL, RTOL = 1e-4, 1e-3


def _engine(builder, tmp_path, **kw):
    from fxfusion_b200.engine import ExecutionEngine
    graph = builder.finish()
    path = tmp_path / f"{graph.name}.bin"
    wire.dump(graph, path)
    return graph, ExecutionEngine(str(path), "cuda:0", **kw)


def _w(rng, n, k):
    return (rng.standard_normal((n, k), dtype=np.float32) / math.sqrt(k)).astype(np.float32)


# one shape per tile variant and then its edges: one row / column past a tile, K past a 64-deep slab, K-split last rounds,
# outputs without 16-byte rows, a single column
@pytest.mark.parametrize("M,N,K,variant", [
    (8192, 2304, 768, "256x"), (8192, 768, 3072, "256x"), (985, 768, 768, "256x64-pair"), (16384, 512, 512, "256x128-pair"), (8192, 3072, 768, "256x192-pair"),
    (65, 512, 512, "128x32"), (512, 1000, 256, "128x32"), (129, 33, 72, "128x"), (257, 129, 1096, ""), (300, 10, 512, "128x32"), (985, 1111, 264, ""), (66, 1, 16, ""), (513, 50257, 40, "")])
def test_every_variant_at_its_edges(built_lib, tmp_path, M, N, K, variant):
    rng = np.random.default_rng(M + N + K)
    b = lowering.GraphBuilder(f"f16_{M}_{N}_{K}")
    x = b.input((M, K), wire.DT_F32)
    b.output(b.op("LinearRelu", [x, b.const(_w(rng, N, K)), b.const(rng.standard_normal(N, dtype=np.float32))], (M, N)))
    graph, eng = _engine(b, tmp_path)
    assert "split operands: tcgen05-f16x3-" + variant in eng.describe(), eng.describe()
    xin = torch.randn(M, K, generator=torch.Generator().manual_seed(1))
    ok, info = compare_outputs(eng.run([xin.cuda()])[0].cpu(), GraphOracle(graph).run([xin])[0], atol=ATOL, rtol=RTOL)
    assert ok, info
    assert eng.device_status() == 0
    eng.close()


def test_rows_keep_their_precision_at_any_scale(built_lib, tmp_path):
    """Every row carries its own power-of-two scale: rows of 1e-30 and of 1e30 come out as accurately as rows of 1, weight
    rows likewise, a row of zeros gives the bias, and elements 2^-16 of their row's maximum
    keep their own precision."""
    M, N, K = 130, 72, 200
    rng = np.random.default_rng(7)
    w = _w(rng, N, K) * (10.0 ** rng.integers(-6, 6, size=(N, 1))).astype(np.float32)
    w[:, 0] = 0.0
    b = lowering.GraphBuilder("f16_scales")
    x = b.input((M, K), wire.DT_F32)
    b.output(b.op("Linear", [x, b.const(w), b.const(np.zeros(N, np.float32))], (M, N)))
    _, eng = _engine(b, tmp_path)
    xin = torch.randn(M, K, generator=torch.Generator().manual_seed(2)) * 10.0 ** torch.linspace(-30, 30, M).unsqueeze(1)
    xin[5] = 0.0
    xin[6] *= 2.0 ** -16 / xin[6].abs().max()
    xin[6, 0] = 1.0        # meets a zero weight: it sets the row's scale and nothing else
    w64 = torch.from_numpy(w).double()
    want = xin.double() @ w64.T
    scale = xin.double().abs() @ w64.abs().T
    got = eng.run([xin.cuda()])[0].cpu().double()
    assert torch.equal(got[5], torch.zeros(N, dtype=torch.float64))
    ok = scale > 0
    assert ((got - want).abs()[ok] / scale[ok]).max().item() < 2e-6
    eng.close()


# Distance from fp64 (2-norm): both factors to 22 bits and more with lo·lo dropped, 2^-23 together, and `adds` additions to a running
# sum, each truncated by half an ulp, 2^-24, of a sum that is half of the result on average.  Few rows: one addition per 16 elements
# of a slab; else three per 16 elements of a chain of 256 (tiles of up to 64 columns), 512 (128 columns) or 128 (weights streamed).
@pytest.mark.parametrize("M,N,K,adds", [(1, 512, 512, 4), (17, 640, 64, 4), (32, 768, 768, 4), (32, 768, 3072, 4), (64, 1024, 256, 4),
                                        (65, 512, 512, 48), (300, 768, 3072, 48), (1565, 1024, 1024, 96), (40, 19000, 768, 24)])
def test_distance_from_fp64(built_lib, tmp_path, M, N, K, adds):
    rng = np.random.default_rng(M + N + K)
    w = _w(rng, N, K)
    b = lowering.GraphBuilder(f"fp64_{M}_{N}_{K}")
    x = b.input((M, K), wire.DT_F32)
    b.output(b.op("Linear", [x, b.const(w), b.const(np.zeros(N, np.float32))], (M, N)))
    _, eng = _engine(b, tmp_path)
    xin = torch.randn(M, K, generator=torch.Generator().manual_seed(1))
    want = xin.double() @ torch.from_numpy(w).double().T
    got = eng.run([xin.cuda()])[0].cpu().double()
    assert ((got - want).norm() / want.norm()).item() < 2.0 ** -23 + adds * 2.0 ** -25
    eng.close()


@pytest.mark.parametrize("M,D,F", [(65, 64, 256), (200, 768, 3072), (333, 136, 72)])
@pytest.mark.parametrize("precision", ["auto", "bf16"])
def test_activations_stay_in_split_form_between_nodes(built_lib, tmp_path, M, D, F, precision):
    """LayerNorm -> FeedForward and LinearRelu -> LinearRelu -> Linear: the activation between two products is written in
    split form by its producer; one that anything else reads (the second LayerNorm's residual) stays fp32."""
    rng = np.random.default_rng(M)
    b = lowering.GraphBuilder(f"f16_chain_{M}_{D}")
    c = lambda n, k: (b.const(_w(rng, n, k)), b.const(rng.standard_normal(n, dtype=np.float32)))
    x = b.input((M, D), wire.DT_F32)
    ln = b.op("LayerNorm", [x, b.const(rng.standard_normal(D, dtype=np.float32)), b.const(rng.standard_normal(D, dtype=np.float32))], (M, D), ints=[1, D], floats=[1e-5])
    ff = b.op("FeedForward", [ln, *c(F, D), *c(D, F)], (M, D))
    add = b.op("Add", [x, ff], (M, D))
    ln2 = b.op("LayerNorm", [add, b.const(np.ones(D, np.float32)), b.const(np.zeros(D, np.float32))], (M, D), ints=[1, D], floats=[1e-5])
    h1 = b.op("LinearRelu", [ln2, *c(F, D)], (M, F))
    h2 = b.op("LinearRelu", [h1, *c(D, F)], (M, D))
    both = b.op("Add", [h2, ln2], (M, D))
    b.output(b.op("Linear", [both, *c(40, D)], (M, 40)))
    graph, eng = _engine(b, tmp_path, precision=precision)
    text = eng.describe().splitlines()
    split = [("output in split form" in t) for t in text if t.split()[1:2] and t.split()[1] in ("LayerNorm", "LinearRelu")]
    assert split == [True, False, True, False], "\n".join(text)
    xin = torch.randn(M, D, generator=torch.Generator().manual_seed(3))
    got, want = eng.run([xin.cuda()])[0].cpu(), GraphOracle(graph).run([xin])[0]
    if precision == "auto":
        ok, info = compare_outputs(got, want, atol=ATOL * 5, rtol=RTOL)
        assert ok, info
    else:
        assert ((got - want).abs().max() / want.abs().max()).item() < 2e-2
    assert eng.device_status() == 0
    eng.close()


# the few-row kernels: row groups of 16 and 32, clusters of 1 to 16 CTAs over K, several rounds of slabs, a ragged K and N, and
# the streaming kernel for weights of a tile per SM
@pytest.mark.parametrize("M,N,K,variant", [
    (1, 512, 512, "rows128"), (16, 129, 72, "rows128"), (17, 10, 512, "rows128"), (32, 768, 3072, "rows128"), (33, 127, 16, "rows128"), (64, 2304, 768, "rows128"),
    (5, 1, 5000, "rows128"), (64, 512, 8200, "rows128"), (31, 12800, 264, "rows128"), (32, 18945, 768, "stream128"), (33, 19000, 520, "stream128"), (1, 50257, 768, "stream128")])
def test_few_rows(built_lib, tmp_path, M, N, K, variant):
    rng = np.random.default_rng(M + N + K)
    b = lowering.GraphBuilder(f"rows_{M}_{N}_{K}")
    x = b.input((M, K), wire.DT_F32)
    r = b.input((M, N), wire.DT_F32)
    lin = b.op("Linear", [x, b.const(_w(rng, N, K)), b.const(rng.standard_normal(N, dtype=np.float32))], (M, N))
    b.output(b.op("AddRelu", [lin, r], (M, N)))
    graph, eng = _engine(b, tmp_path)
    assert "split operands: tcgen05-f16x3-" + variant in eng.describe() and "+AddRelu(residual" in eng.describe(), eng.describe()
    gen = torch.Generator().manual_seed(1)
    xin, rin = torch.randn(M, K, generator=gen), torch.randn(M, N, generator=gen)
    xin *= 10.0 ** torch.linspace(-6, 6, K)   # K ranges of very different size: every CTA of a cluster scales its own
    got, want = eng.run([xin.cuda(), rin.cuda()])[0].cpu(), GraphOracle(graph).run([xin, rin])[0]
    assert ((got - want).abs().max() / want.abs().max()).item() < 2e-6
    xin = torch.randn(M, K, generator=gen)
    ok, info = compare_outputs(eng.run([xin.cuda(), rin.cuda()])[0].cpu(), GraphOracle(graph).run([xin, rin])[0], atol=2e-5, rtol=1e-4)
    assert ok, info
    assert eng.device_status() == 0
    eng.close()


# cluster sizes between the powers of two (K-slabs divided unevenly, several rounds of them), and grids of more than one wave
@pytest.mark.parametrize("M,N,K", [(32, 2048, 3072), (20, 2944, 3080), (64, 2944, 1536), (3, 1500, 1536), (64, 896, 1000), (2, 8192, 704), (48, 4096, 4096)])
def test_few_rows_of_any_cluster(built_lib, tmp_path, M, N, K):
    test_few_rows(built_lib, tmp_path, M, N, K, "rows128")


# channels-last images in split form: image borders inside a tile (14 x 14, 7 x 7), several images per tile, ragged channels,
# asymmetric filters and padding, strides, dilation, a map of one pixel, and one image of many tiles
@pytest.mark.parametrize("N,size,C,O,kh,kw,s,ph,pw,d", [
    (2, 56, 64, 96, 3, 3, 1, 1, 1, 1), (5, 28, 40, 72, 3, 3, 2, 1, 1, 1), (3, 57, 128, 256, 1, 1, 2, 0, 0, 1), (7, 30, 24, 64, 5, 3, 1, 2, 0, 1), (2, 64, 64, 64, 3, 5, 1, 2, 4, 2),
    (1, 26, 512, 128, 7, 7, 1, 0, 0, 1), (1, 224, 64, 256, 3, 3, 1, 1, 1, 1), (33, 12, 16, 200, 3, 3, 1, 1, 1, 1)])
def test_images_in_split_form(built_lib, tmp_path, N, size, C, O, kh, kw, s, ph, pw, d):
    """Stem, max pooling, convolutions, the residual AddRelu in the epilogue of one of them and global average pooling hand
    the images on in split form; a convolution that feeds a plain average pooling leaves fp32 pixels."""
    rng = np.random.default_rng(size + C)
    gb = [1, 1, 1, 256, 1, 1]
    b = lowering.GraphBuilder(f"images_{N}_{size}_{C}_{O}")

    def conv(x, c, o, h, w, kh=1, kw=1, s=1, ph=0, pw=0, d=1, relu=True):
        ho, wo = (h + 2 * ph - d * (kh - 1) - 1) // s + 1, (w + 2 * pw - d * (kw - 1) - 1) // s + 1
        weight = (rng.standard_normal((o, c, kh, kw)) / math.sqrt(c * kh * kw)).astype(np.float32)
        y = b.op("Conv2dRelu" if relu else "Conv2d", [x, b.const(weight), b.const(rng.standard_normal(o, dtype=np.float32))], (N, o, ho, wo), ints=[s, s, ph, pw, d, d, 1] + gb)
        return y, ho, wo

    x = b.input((N, 3, size, size), wire.DT_F32)
    y, h, w = conv(x, 3, 64, size, size, 7, 7, 2, 3, 3)
    h, w = (h - 1) // 2 + 1, (w - 1) // 2 + 1
    y = b.op("MaxPool2d", [y], (N, 64, h, w), ints=[3, 3, 2, 2, 1, 1, 1, 1, 0] + gb)
    y, h, w = conv(y, 64, C, h, w)
    r, _, _ = conv(y, C, 2 * O, h, w, kh, kw, s, ph, pw, d, relu=False)
    y, h, w = conv(y, C, O, h, w, kh, kw, s, ph, pw, d)
    y, _, _ = conv(y, O, 2 * O, h, w, relu=False)
    y = b.op("AddRelu", [y, r], (N, 2 * O, h, w))
    z, _, _ = conv(y, 2 * O, 24, h, w)
    z = b.op("AvgPool2d", [z], (N, 24, h, w), ints=[1, 1, 1, 1, 0, 0, 0] + gb)
    b.output(conv(z, 24, 8, h, w)[0])
    b.output(b.op("AdaptiveAvgPool2d", [y], (N, 2 * O, 1, 1), ints=[1, 1] + gb))
    graph, eng = _engine(b, tmp_path)
    text = eng.describe()
    assert text.count("images in split form") == 6 and text.count("output in split form") == 6 and "+AddRelu(residual" in text, text
    xin = torch.randn(N, 3, size, size, generator=torch.Generator().manual_seed(3)) * 10.0 ** torch.linspace(-8, 8, N).reshape(N, 1, 1, 1)
    got, want = eng.run([xin.cuda()]), GraphOracle(graph).run([xin])
    for g, t in zip(got, want):
        scale = t.abs().amax(dim=(1, 2, 3), keepdim=True)
        assert ((g.cpu() - t).abs() / scale).max().item() < 4e-6
    eng.run([xin.cuda() * 1e-3])   # the maxima of one forward do not stay for the next
    again = eng.run([xin.cuda()])
    assert all(torch.equal(a.cpu(), g.cpu()) for a, g in zip(again, got))
    assert eng.device_status() == 0
    eng.close()


@pytest.mark.parametrize("B,T,D,P,lead", [(2, 5, 64, 9, 0), (3, 7, 30, 7, 2), (1, 1, 4, 1, 0)])
def test_embedding_scale_add_is_one_pass(built_lib, tmp_path, B, T, D, P, lead):
    """Embedding -> Mul -> Add of a slice of a positional table: one launch with the roundings of the separate nodes; an index
    outside the table still sets the status."""
    rng = np.random.default_rng(T)
    b = lowering.GraphBuilder(f"emb_{B}_{T}_{D}")
    ids = b.input((B, T), wire.DT_I64)
    mul = b.op("Mul", [b.op("Embedding", [ids, b.const(rng.standard_normal((11, D), dtype=np.float32))], (B, T, D))], (B, T, D), ints=[1], floats=[math.sqrt(D)])
    size = b.op("Size", [mul], (), wire.DT_I64, ints=[1])
    nar = b.op("Narrow", [b.const(rng.standard_normal((1, P + lead, D), dtype=np.float32)), size], (1, T, D), ints=[1, lead, -1])
    b.output(b.op("Add", [mul, nar], (B, T, D)))
    graph, eng = _engine(b, tmp_path)
    x = torch.randint(0, 11, (B, T), generator=torch.Generator().manual_seed(0))
    assert torch.equal(eng.run([x.cuda()])[0].cpu(), GraphOracle(graph).run([x])[0])
    eng.profile_launches()
    assert len(eng.profile_launches()) == 1
    assert eng.device_status() == 0
    x[0, 0] = 11
    eng.run([x.cuda()])
    assert eng.device_status() != 0
    eng.close()


@pytest.mark.parametrize("N,O,chunk", [(81, 1024, 512), (81, 1024, 0), (20, 1024, 1024)])
def test_short_convolutions_with_long_chains(built_lib, tmp_path, N, O, chunk):
    """1x1 convolutions of 14 x 14 images, 512 channels: with chains as long as their depth they run with sixteen epilogue warps
    and cut tiles along K (fxf_gemm_workspace: 1920 flags at 81 images), residual and maxima included."""
    from fxfusion_b200.kernels import gemm_workspace
    cut = gemm_workspace(N * 196, O, 512, images=True, tc_chunk_k=chunk)
    assert cut["flags"] <= cut["flags_kept"] and (chunk != 512 or cut["flags"] == 1920)
    rng = np.random.default_rng(N)
    gb = [1, 1, 1, 256, 1, 1]
    b = lowering.GraphBuilder(f"cut_{N}_{O}_{chunk}")

    def conv(x, c, o, k, s, p, h, relu=True):
        w = (rng.standard_normal((o, c, k, k)) / math.sqrt(c * k * k)).astype(np.float32)
        return b.op("Conv2dRelu" if relu else "Conv2d", [x, b.const(w), b.const(rng.standard_normal(o, dtype=np.float32))], (N, o, h, h), ints=[s, s, p, p, 1, 1, 1] + gb)

    x = b.input((N, 3, 28, 28), wire.DT_F32)
    y = conv(x, 3, 512, 7, 2, 3, 14)
    r = conv(y, 512, O, 1, 1, 0, 14, relu=False)
    y = b.op("AddRelu", [conv(y, 512, O, 1, 1, 0, 14, relu=False), r], (N, O, 14, 14))
    y = conv(y, O, 512, 1, 1, 0, 14)
    b.output(b.op("AdaptiveAvgPool2d", [y], (N, 512, 1, 1), ints=[1, 1] + gb))
    graph, eng = _engine(b, tmp_path, tc_chunk_k=chunk)
    assert eng.describe().count("output in split form") == 4, eng.describe()
    xin = torch.randn(N, 3, 28, 28, generator=torch.Generator().manual_seed(5))
    want = GraphOracle(graph).run([xin])[0]
    for _ in range(3):   # the flags are zero again after every launch
        got = eng.run([xin.cuda()])[0].cpu()
        assert ((got - want).abs().max() / want.abs().max()).item() < (4e-6 if chunk == 0 else 4e-5)
    assert eng.device_status() == 0
    eng.close()


@pytest.mark.parametrize("pad_x,pad_y", [(0, 0), (12, 0), (0, 4), (12, 4)])
def test_rows_at_any_offset(built_lib, tmp_path, pad_x, pad_y):
    """A graph file may place activations at any multiple of four bytes: where a LayerNorm, its input, its weights (a slice of a
    constant) or a product's result does not lie on a 16-byte address, the rows stay fp32 and the results are the same."""
    M, D, F = 70, 64, 96
    rng = np.random.default_rng(1)
    b = lowering.GraphBuilder(f"offsets_{pad_x}_{pad_y}", alignment=4)
    c = lambda n, k: (b.const(_w(rng, n, k)), b.const(rng.standard_normal(n, dtype=np.float32)))
    pads = []

    def pad(nbytes):   # an activation that lives to the end, so that what follows lies `nbytes` further on
        if nbytes:
            pads.append(b.op("Relu", [b.input((nbytes // 4,), wire.DT_F32)], (nbytes // 4,)))

    def slice_from(lead):   # a slice of a constant, `lead` floats behind its begin
        return b.op("Narrow", [b.const(rng.standard_normal(D + 4, dtype=np.float32))], (D,), ints=[0, lead, D])

    x0 = b.input((M, D), wire.DT_F32)
    pad(pad_x)
    x = b.op("Relu", [x0], (M, D))
    pad(pad_y)
    ln = b.op("LayerNorm", [x, slice_from(4), slice_from(0)], (M, D), ints=[1, D], floats=[1e-5])
    ln2 = b.op("LayerNorm", [x, slice_from(1), slice_from(0)], (M, D), ints=[1, D], floats=[1e-5])   # never: its weights lie on 4 bytes
    h = b.op("LinearRelu", [ln, *c(F, D)], (M, F))
    g = b.op("FeedForward", [ln2, *c(F, D), *c(D, F)], (M, D))
    h2 = b.op("Linear", [h, *c(D, F)], (M, D))
    b.output(b.op("Add", [h2, g], (M, D)))
    for p in pads:
        b.output(p)
    graph, eng = _engine(b, tmp_path)
    text = eng.describe().splitlines()
    split = [("output in split form" in t) for t in text if t.split()[1:2] and t.split()[1] in ("LayerNorm", "LinearRelu")]
    assert split == [pad_x == 0 and pad_y == 0, False, (pad_x + pad_y) % 16 == 0], "\n".join(text)
    gen = torch.Generator().manual_seed(3)
    xin = [torch.randn(M, D, generator=gen)] + [torch.randn(n // 4, generator=gen) for n in (pad_x, pad_y) if n]
    got, want = eng.run([t.cuda() for t in xin]), GraphOracle(graph).run(xin)
    for o, w in zip(got, want):
        ok, info = compare_outputs(o.cpu(), w, atol=ATOL, rtol=RTOL)
        assert ok, info
    assert eng.device_status() == 0
    eng.close()


@pytest.mark.parametrize("pad,later", [(0, False), (4, False), (12, False), (8, True)])
def test_images_at_any_offset(built_lib, tmp_path, pad, later):
    """The same for images: what does not lie on a 16-byte address is kept as fp32 pixels (`later`: from the second convolution's
    result on), whatever its neighbours could do."""
    N, rng, gb = 3, np.random.default_rng(2), [1, 1, 1, 256, 1, 1]
    b = lowering.GraphBuilder(f"image_offsets_{pad}_{later}", alignment=4)

    def conv(x, c, o, h, k, s, p, relu=True):
        ho = (h + 2 * p - k) // s + 1
        w = (rng.standard_normal((o, c, k, k)) / math.sqrt(c * k * k)).astype(np.float32)
        return b.op("Conv2dRelu" if relu else "Conv2d", [x, b.const(w), b.const(rng.standard_normal(o, dtype=np.float32))], (N, o, ho, ho), ints=[s, s, p, p, 1, 1, 1] + gb)

    x = b.input((N, 3, 48, 48), wire.DT_F32)
    odd = b.input((pad // 4,), wire.DT_F32) if pad else None
    keep = b.op("Relu", [odd], (pad // 4,)) if pad and not later else None
    y = b.op("MaxPool2d", [conv(x, 3, 64, 48, 7, 2, 3)], (N, 64, 12, 12), ints=[3, 3, 2, 2, 1, 1, 1, 1, 0] + gb)
    r = conv(y, 64, 128, 12, 1, 1, 0, relu=False)
    if pad and later:
        keep = b.op("Relu", [odd], (pad // 4,))
    t = conv(y, 64, 64, 12, 3, 1, 1)
    y = b.op("AddRelu", [conv(t, 64, 128, 12, 1, 1, 0, relu=False), r], (N, 128, 12, 12))
    b.output(b.op("AdaptiveAvgPool2d", [conv(y, 128, 72, 12, 3, 2, 1)], (N, 72, 1, 1), ints=[1, 1] + gb))
    if keep is not None:
        b.output(keep)
    graph, eng = _engine(b, tmp_path)
    count = eng.describe().count("output in split form")
    assert count == 6 if pad == 0 else (count == 0 if not later else count < 6), eng.describe()
    gen = torch.Generator().manual_seed(4)
    xin = [torch.randn(N, 3, 48, 48, generator=gen)] + ([torch.randn(pad // 4, generator=gen)] if pad else [])
    got, want = eng.run([t.cuda() for t in xin]), GraphOracle(graph).run(xin)
    assert ((got[0].cpu() - want[0]).abs().max() / want[0].abs().max()).item() < 4e-6
    assert eng.device_status() == 0
    eng.close()


@pytest.mark.parametrize("M,precision", [(1, "auto"), (32, "auto"), (70, "auto"), (300, "auto"), (70, "fp32_3xtf32"), (70, "bf16")])
@pytest.mark.parametrize("what", ["weight", "bias", "both"])
def test_weights_that_are_not_constants(built_lib, tmp_path, M, what, precision):
    """Only constants are converted at build time: a weight or bias that is an input of the graph, or computed by the node
    before, is read when the product runs."""
    K, N = 72, 136
    rng = np.random.default_rng(M)
    b = lowering.GraphBuilder(f"live_{M}_{what}")
    x = b.input((M, K), wire.DT_F32)
    w1, w2, b1, b2 = _w(rng, N, K), _w(rng, K, N), rng.standard_normal(N, dtype=np.float32), rng.standard_normal(K, dtype=np.float32)
    given = []

    def weight(a):
        if what == "bias":
            return b.const(a)
        given.append(a)
        return b.input(a.shape, wire.DT_F32)

    def bias(a):
        if what == "weight":
            return b.const(a)
        given.append(a)
        return b.op("Mul", [b.input(a.shape, wire.DT_F32)], a.shape, ints=[1], floats=[2.0])

    ff = [weight(w1), bias(b1), weight(w2), bias(b2)]
    y = b.op("FeedForward", [x, *ff], (M, K))
    y = b.op("LinearRelu", [y, ff[0], ff[1]], (M, N))
    b.output(b.op("Linear", [y, b.const(w2), bias(b2) if what != "weight" else b.const(b2)], (M, K)))
    graph, eng = _engine(b, tmp_path, precision=precision)
    gen = torch.Generator().manual_seed(1)
    for scale in (1.0, 3.0):   # the second run brings other weights
        xin = [torch.randn(M, K, generator=gen)] + [torch.from_numpy(a * np.float32(scale)) for a in given]
        got, want = eng.run([t.cuda() for t in xin])[0].cpu(), GraphOracle(graph).run(xin)[0]
        if precision == "bf16":   # where weights are constants their products round both factors to bf16
            assert ((got - want).abs().max() / want.abs().max()).item() < 2e-2
            continue
        ok, info = compare_outputs(got, want, atol=1e-3, rtol=1e-3)
        assert ok, info
    assert eng.device_status() == 0
    eng.close()


def test_filters_that_are_not_constants(built_lib, tmp_path):
    """A convolution between images in split form whose filters are an input of the graph: it reads them when it runs, and its
    neighbours keep the images it touches as fp32 pixels."""
    N, rng, gb = 2, np.random.default_rng(3), [1, 1, 1, 256, 1, 1]
    b = lowering.GraphBuilder("live_filters")
    w = lambda o, c, k: (rng.standard_normal((o, c, k, k)) / math.sqrt(c * k * k)).astype(np.float32)
    bias = lambda o: b.const(rng.standard_normal(o, dtype=np.float32))
    x = b.input((N, 3, 32, 32), wire.DT_F32)
    y = b.op("Conv2dRelu", [x, b.const(w(64, 3, 7)), bias(64)], (N, 64, 16, 16), ints=[2, 2, 3, 3, 1, 1, 1] + gb)
    y = b.op("Conv2dRelu", [y, b.const(w(64, 64, 3)), bias(64)], (N, 64, 16, 16), ints=[1, 1, 1, 1, 1, 1, 1] + gb)
    live = w(128, 64, 3)
    y = b.op("Conv2dRelu", [y, b.input(live.shape, wire.DT_F32), bias(128)], (N, 128, 16, 16), ints=[1, 1, 1, 1, 1, 1, 1] + gb)
    y = b.op("Conv2dRelu", [y, b.input((64, 128, 1, 1), wire.DT_F32), bias(64)], (N, 64, 16, 16), ints=[1, 1, 0, 0, 1, 1, 1] + gb)
    b.output(b.op("AdaptiveAvgPool2d", [y], (N, 64, 1, 1), ints=[1, 1] + gb))
    graph, eng = _engine(b, tmp_path)
    assert eng.describe().count("output in split form") == 1, eng.describe()
    gen = torch.Generator().manual_seed(1)
    for scale in (1.0, 2.0):
        xin = [torch.randn(N, 3, 32, 32, generator=gen), torch.from_numpy(live * np.float32(scale)), torch.from_numpy(w(64, 128, 1))]
        ok, info = compare_outputs(eng.run([t.cuda() for t in xin])[0].cpu(), GraphOracle(graph).run(xin)[0], atol=ATOL, rtol=RTOL)
        assert ok, info
    assert eng.device_status() == 0
    eng.close()


@pytest.mark.parametrize("dim,refused", [(1, False), (-2, False), (3, True), (-4, True)])
def test_size_that_nothing_needs_is_still_checked(built_lib, tmp_path, dim, refused):
    """A Size read only by the Narrow of a constant launches nothing, and is refused as before where its dimension does not exist."""
    b = lowering.GraphBuilder(f"size_{dim}")
    x = b.input((2, 5, 8), wire.DT_F32)
    y = b.op("Relu", [x], (2, 5, 8))
    size = b.op("Size", [y], (), wire.DT_I64, ints=[dim])
    table = np.random.default_rng(0).standard_normal((1, 9, 8), dtype=np.float32)
    b.output(b.op("Add", [y, b.op("Narrow", [b.const(table), size], (1, 5, 8), ints=[1, 0, -1])], (2, 5, 8)))
    if refused:
        with pytest.raises(RuntimeError, match="size: dim out of range"):
            _engine(b, tmp_path)
        return
    graph, eng = _engine(b, tmp_path)
    xin = torch.randn(2, 5, 8)
    assert torch.equal(eng.run([xin.cuda()])[0].cpu(), GraphOracle(graph).run([xin])[0])
    eng.close()


@pytest.mark.parametrize("op", ["LayerNorm", "AddLayerNorm"])
def test_rows_normalised_in_place_stay_fp32(built_lib, tmp_path, op):
    """A file may place a LayerNorm's result on its input.  Row by row that works in fp32; in split form the planes of a row would
    cover rows that other blocks have not read yet."""
    from fxfusion_b200.engine import ExecutionEngine
    M, D = 3000, 128
    rng = np.random.default_rng(5)
    b = lowering.GraphBuilder(f"in_place_{op}")
    x = b.op("Relu", [b.input((M, D), wire.DT_F32)], (M, D))
    affine = [b.const(rng.standard_normal(D, dtype=np.float32)), b.const(rng.standard_normal(D, dtype=np.float32))]
    ln = b.op(op, ([x] if op == "LayerNorm" else [x, b.input((M, D), wire.DT_F32)]) + affine, (M, D), ints=[1, D], floats=[1e-5])
    b.output(b.op("Linear", [ln, b.const(_w(rng, 64, D)), b.const(np.zeros(64, np.float32))], (M, 64)))
    graph = b.finish()
    want_graph = graph.tensors[ln].offset
    gen = torch.Generator().manual_seed(1)
    xin = [torch.randn(M, D, generator=gen) for _ in range(1 if op == "LayerNorm" else 2)]
    want = GraphOracle(graph).run(xin)[0]
    graph.tensors[ln].offset = graph.tensors[x].offset
    assert graph.tensors[ln].offset != want_graph
    wire.dump(graph, tmp_path / "g.bin")
    eng = ExecutionEngine(str(tmp_path / "g.bin"), "cuda:0")
    assert "output in split form" not in eng.describe()
    ok, info = compare_outputs(eng.run([t.cuda() for t in xin])[0].cpu(), want, atol=ATOL, rtol=RTOL)
    assert ok, info
    eng.close()


@pytest.mark.parametrize("precision", ["auto", "fp32_tf32_bf16x2"])
@pytest.mark.parametrize("form", ["rows", "few rows", "images"])
def test_dynamic_range_inside_a_row_and_an_image(built_lib, tmp_path, form, precision):
    """Columns of a row (channels of an image) from 1 down to 2^-44 of the largest, each scaled back up by the next product.  In split
    form an element has 22 bits or an absolute error of 2^-39 of its row's (image's) bound, whichever is coarser, where the bound is
    max|x| * max ||w||_1 + max|b|; the TF32 arithmetic keeps an exponent per element."""
    C, size = 48, 16
    rng = np.random.default_rng(9)
    shrink = 2.0 ** -np.arange(C, dtype=np.float32)
    shrink[shrink < 2.0 ** -44] = 2.0 ** -44
    # weights of one sign on inputs that a ReLU made: no column is small by cancellation
    w1 = (np.abs(rng.standard_normal((C, 64), dtype=np.float32)) * shrink[:, None]).astype(np.float32)
    w2 = np.diag(1.0 / shrink).astype(np.float32)
    zero = np.zeros(C, np.float32)
    gen = torch.Generator().manual_seed(1)
    b = lowering.GraphBuilder(f"range_{form.split()[0]}_{precision}")
    if form == "images":
        N, gb = 3, [1, 1, 1, 256, 1, 1]
        x = b.input((N, 3, 2 * size, 2 * size), wire.DT_F32)
        conv = lambda op, t, w, bias, k, s, p: b.op(op, [t, b.const(w), b.const(bias)], (N, w.shape[0], size, size), ints=[s, s, p, p, 1, 1, 1] + gb)
        y = conv("Conv2dRelu", x, (rng.standard_normal((64, 3, 7, 7)) / 12).astype(np.float32), rng.standard_normal(64, dtype=np.float32), 7, 2, 3)
        h = conv("Conv2dRelu", y, w1.reshape(C, 64, 1, 1), zero, 1, 1, 0)
        out = conv("Conv2d", h, w2.reshape(C, C, 1, 1), zero, 1, 1, 0)
        b.output(b.op("AvgPool2d", [out], (N, C, size, size), ints=[1, 1, 1, 1, 0, 0, 0] + gb))
        xin = torch.randn(N, 3, 2 * size, 2 * size, generator=gen)
    else:
        M = 300 if form == "rows" else 40
        x = b.input((M, 64), wire.DT_F32)
        y = b.op("Relu", [x], (M, 64))
        h = b.op("LinearRelu", [y, b.const(w1), b.const(zero)], (M, C))
        b.output(b.op("Linear", [h, b.const(w2), b.const(zero)], (M, C)))
        xin = torch.randn(M, 64, generator=gen)
    graph, eng = _engine(b, tmp_path, precision=precision)
    oracle = GraphOracle(graph)
    want = oracle.run([xin])[0].double()
    bound = oracle.reg[y].abs().max().item() * np.abs(w1).sum(1).max()
    got = eng.run([xin.cuda()])[0].cpu().double()
    dims = (0, 2, 3) if form == "images" else (0,)
    err, top = (got - want).abs().amax(dim=dims), want.abs().amax(dim=dims)
    lost = 2.0 ** -39 * bound / torch.from_numpy(shrink).double() if precision == "auto" else torch.zeros(C, dtype=torch.float64)
    assert (err <= 4e-6 * top + lost).all(), (err / top, lost)
    assert (err[:20] <= 4e-6 * top[:20]).all()   # to 2^-19 of the largest nothing shows
    eng.close()
