"""Sizes at which the kernels' splits have an edge: remainders of tiles and units, the smallest and largest of a
range, addresses with the least alignment that an entry point takes."""

import numpy as np
import pytest
import torch

import tensor_b200 as tb
from oracle import gguf_oracle as oracle

pytestmark = pytest.mark.gpu
FORMATS = ("q8_0", "q4_0", "q4_k", "q6_k")


def dev():
    return torch.device("cuda", 0)


def to_dev(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).to(dev())
    return t if dtype is None else t.to(dtype)


@pytest.fixture(scope="module", autouse=True)
def _no_device_timeouts():
    yield
    assert tb.device_status() == 0


# ---- dequantisation: units of 256 weights, four per warp and step ------------------------------------------------

@pytest.mark.parametrize("offset", [0, 2])
@pytest.mark.parametrize("name", FORMATS)
def test_dequant_partial_units_and_two_byte_alignment(name, offset):
    step = tb.get_format(name).weights
    for n, k in [(1, step), (3, 3 * step), (5, 37 * step), (1031, 7 * step)]:
        raw = oracle.make_weights(name, n, k, seed=n + k)
        buf = torch.zeros(raw.size + 16, dtype=torch.uint8, device=dev())
        buf[offset:offset + raw.size] = to_dev(raw)
        out = torch.full((n, k), float("nan"), device=dev())
        tb.dequantize(buf[offset:offset + raw.size], name, n, k, out=out)
        want = oracle.dequantize(raw, name, n, k)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))


# ---- prefill GEMM: pairs of CTAs, 256 weight rows x 32 .. 256 tokens, 64-wide k-blocks, K split over 1, 2 or 4 pairs --

@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("m,n,blocks", [
    (1, 1, 1), (17, 127, 3), (32, 257, 5), (33, 300, 8), (64, 256, 16), (130, 129, 9), (256, 513, 7), (257, 384, 12),
    (300, 1031, 17), (513, 260, 24),
])
def test_gemm_pair_edges(name, m, n, blocks):
    # blocks counts 256 weights for the K-quants and 32 for the others: k-blocks and raw chunks with every remainder,
    # rows of every 2-byte alignment
    k = blocks * tb.get_format(name).weights * (1 if tb.get_format(name).weights == 256 else 5)
    raw = oracle.make_weights(name, n, k, seed=n + k)
    x = oracle.make_activations(m, k, seed=m, dtype="bf16")
    out = torch.full((m, n), float("nan"), device=dev())
    tb.gemm(to_dev(x, torch.bfloat16), to_dev(raw), name, n, k, out=out)
    want = oracle.gemm_ref(x, raw, name, n, k, operand="bf16")
    # bf16 operands are the same bits on both sides; fp32 sums of K <= 6144 products of random sign differ by a few
    # times sqrt(K) 2^-24 = 4.7e-6 of the result
    assert oracle.rel_frobenius(out.cpu().numpy(), want) < 2e-5


@pytest.mark.parametrize("name,m,n,k", [("q4_k", 600, 12300, 512), ("q6_k", 600, 12300, 768), ("q6_k", 520, 17000, 256),
                                        ("q8_0", 700, 11000, 544), ("q4_0", 700, 11000, 352), ("q8_0", 903, 20160, 544),
                                        ("q4_0", 494, 11583, 4288)])
def test_gemm_pair_several_tiles_per_pair(name, m, n, k):
    """More tiles than pairs: accumulator sets, stages and raw chunks go round."""
    raw = oracle.make_weights(name, n, k, seed=3)
    x = oracle.make_activations(m, k, seed=4, dtype="bf16")
    xd, wd = to_dev(x, torch.bfloat16), to_dev(raw)
    out = torch.full((m, n), float("nan"), device=dev())
    tb.gemm(xd, wd, name, n, k, out=out)
    w = tb.dequantize(wd, name, n, k).to(torch.bfloat16).double()
    want = xd.double() @ w.t()
    assert float((out.double() - want).norm() / want.norm()) < 2e-5  # as above
    again = torch.full((m, n), float("nan"), device=dev())
    tb.gemm(xd, wd, name, n, k, out=again)
    assert torch.equal(out, again)


@pytest.mark.parametrize("name", ["q8_0", "q4_0"])
@pytest.mark.parametrize("m,n,k", [(17, 300, 512), (64, 129, 544), (65, 512, 4096), (130, 257, 7936), (333, 9728, 2048),
                                   (40, 256, 28672), (100, 300, 64), (20, 100, 32)])
def test_gemm_of_32_weight_blocks_sums_in_fp32(name, m, n, k):
    """These formats' prompts are added up outside the tensor cores, which truncate when they accumulate."""
    wd = to_dev(oracle.make_weights(name, n, k, seed=k))
    x = to_dev(oracle.make_activations(m, k, seed=m, dtype="bf16"), torch.bfloat16)
    out = torch.full((m, n), float("nan"), device=dev())
    tb.gemm(x, wd, name, n, k, out=out)
    want = x.double() @ tb.dequantize(wd, name, n, k).to(torch.bfloat16).double().t()
    # four truncating steps of at most 2^-24 = 6e-8 of the sum each, and fp32 additions of 8 and of up to 56 such sums
    # (a few 2^-24, random); accumulated over all of K in the tensor cores the error is 1e-6 at K = 2048
    assert float((out.double() - want).norm() / want.norm()) < 3e-7


@pytest.mark.parametrize("m,n,k", [(9, 777, 4352), (3, 257, 18944), (15, 129, 12288)])
def test_split_gemv_with_odd_row_counts(m, n, k):
    """K split over CTAs with an odd number of partial sums: what lies behind them in the scratch stays aligned."""
    raw = oracle.make_weights("q4_k", n, k, seed=61)
    x = oracle.make_activations(m, k, seed=62, dtype="bf16")
    out = torch.full((m, n), float("nan"), device=dev())
    tb.gguf(m, n, k, "q4_k", variant="fast").launch(to_dev(x, torch.bfloat16), to_dev(raw), out)
    assert oracle.rel_frobenius(out.cpu().numpy(), oracle.gemv_ref(x, raw, "q4_k", n, k)) < 2e-5
    assert tb.device_status() == 0


# ---- decode GEMV with activations in registers: slices of 256, 16 slices a CTA, clusters along K, tiles of 16 rows ----

@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("m,n,blocks,x", [
    (2, 1, 1, "bf16"), (3, 15, 2, "f16"), (8, 17, 9, "bf16"), (9, 100, 5, "bf16"), (16, 2500, 3, "f16"), (16, 33, 17, "bf16"),
    (5, 513, 33, "bf16"), (7, 20, 112, "bf16"), (1, 31, 16, "f32"), (2, 300, 7, "f32"), (3, 49, 40, "f32"), (16, 64, 11, "f32"),
    (1, 130, 15, "bf16"), (8, 100, 16, "bf16"), (12, 2049, 16, "bf16"),
])
def test_gemv_frag_edges(name, m, n, blocks, x):
    # blocks counts 256 weights for the K-quants and 32 for the others (times 5 where that leaves a part of a slice)
    step = tb.get_format(name).weights
    k = blocks * step if step == 256 else blocks * step * 5
    raw = oracle.make_weights(name, n, k, seed=n + k)
    xs = oracle.make_activations(m, k, seed=m, dtype="f32" if x == "f32" else x)
    dtype = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}[x]
    xd, wd = to_dev(xs, dtype), to_dev(raw)
    kernel = tb.gguf(m, n, k, name, x_dtype=dtype)
    out, again = (torch.full((m, n), float("nan"), device=dev()) for _ in range(2))
    kernel.launch(xd, wd, out)
    kernel.launch(xd, wd, again)
    assert torch.equal(out, again)
    want = xd.double() @ tb.dequantize(wd, name, n, k).double().t()
    # exact operands; fp32 sums of up to 28672 products: a few times sqrt(K) 2^-24 = 1e-5 (Q4_K's own pipeline, which
    # takes its 2-byte activations, loses three bits to the offset of its integers)
    assert float((out.double() - want).norm() / want.norm()) < (2e-5 if name == "q4_k" else 1e-5)


@pytest.mark.parametrize("name,m,n,k,x", [
    ("q8_0", 1, 31, 96, "f32"), ("q8_0", 2, 2000, 512, "f32"), ("q8_0", 1, 4097, 4096, "f32"), ("q8_0", 3, 17, 4096, "f32"),
    ("q8_0", 1, 33, 96, "bf16"), ("q4_0", 1, 31, 96, "f32"), ("q4_0", 16, 100, 8224, "f32"), ("q4_0", 1, 40, 4128, "f16"),
    ("q6_k", 1, 31, 256, "f32"), ("q6_k", 2, 1537, 2048, "f32"), ("q6_k", 1, 130, 12288, "f32"), ("q6_k", 1, 50, 768, "bf16"),
    ("q4_k", 1, 31, 256, "f32"), ("q4_k", 4, 300, 18432, "f32"), ("q4_k", 9, 2100, 3840, "f16"), ("q4_k", 16, 2500, 4352, "f16"),
    ("q4_k", 8, 513, 4096, "f16"), ("q4_k", 5, 4100, 8192, "f16"), ("q4_k", 2, 4097, 12288, "bf16"),
    ("q4_k", 16, 20, 28672, "bf16"), ("q4_k", 16, 33, 32768, "f16"),
])
def test_gemv_frag_shapes_that_run_on_it(name, m, n, k, x):
    """Of the launches that other kernels share, sizes that the default sends to the register kernel."""
    dtype = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}[x]
    assert tb.ops.gemv_on_registers(name, m, n, k, dtype)
    wd = to_dev(oracle.make_weights(name, n, k, seed=n))
    xd = to_dev(oracle.make_activations(m, k, seed=k, dtype=x), dtype)
    out = torch.full((m, n), float("nan"), device=dev())
    tb.gguf(m, n, k, name, x_dtype=dtype).launch(xd, wd, out)
    want = xd.double() @ tb.dequantize(wd, name, n, k).double().t()
    # fp32 sums of 16-slice CTAs: 2.4e-8 sqrt(8 + 4) = 8e-8 at K = 4096, a little more per CTA of a cluster; Q4_K's chains
    # truncate up to 16 times 1.3e-8 besides
    assert float((out.double() - want).norm() / want.norm()) < (1e-6 if name == "q4_k" else 4e-7)


def balanced_q4_k(n, k, seed):
    """Q4_K blocks as a quantised weight of mean zero has them: every group's minimum is 7.5 times its scale."""
    raw = oracle.make_weights("q4_k", n, k, seed=seed).reshape(-1, 144)
    d = np.ascontiguousarray(raw[:, 0:2]).view(np.float16).astype(np.float32)
    raw[:, 2:4] = (7.5 * d).astype(np.float16).view(np.uint8)
    raw[:, 8:12] = raw[:, 4:8]
    raw[:, 12:16] = (raw[:, 12:16] & 15) * 17
    return raw.reshape(-1)


@pytest.mark.parametrize("exponent", [0, -4, -7, -10, -12, -14, -16])
@pytest.mark.parametrize("m,k", [(4, 4096), (16, 4096), (4, 12288), (16, 12288)])
def test_gemv_frag_q4k_small_f16_activations(m, k, exponent):
    """The minimums' share of a result is as large as the quants': group sums keep their precision at every magnitude."""
    n = 272 if k == 4096 else 4112
    assert tb.ops.gemv_on_registers("q4_k", m, n, k, "float16")
    wd = to_dev(balanced_q4_k(n, k, seed=k))
    gen = torch.Generator(device=dev()).manual_seed(m)
    x = (torch.randn((m, k), device=dev(), generator=gen) * 2.0 ** exponent).to(torch.float16)
    x[m - 1, 256:512] = 0
    out = torch.full((m, n), float("nan"), device=dev())
    tb.gguf(m, n, k, "q4_k", x_dtype="float16").launch(x, wd, out)
    want = x.double() @ tb.dequantize(wd, "q4_k", n, k).double().t()
    # exact operands: fp32 sums of up to 12288 products, a few times sqrt(K) 2^-24 = 6.6e-6 of terms about twice the result
    assert float((out.double() - want).norm() / want.norm()) < 2e-5


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("m,n,k", [(1, 4112, 4096), (5, 1024, 4096), (16, 512, 4096), (3, 512, 12288)])
def test_gemv_frag_f32_sums_like_fp32_arithmetic(name, m, n, k):
    wd = to_dev(oracle.make_weights(name, n, k, seed=m))
    x = torch.randn((m, k), device=dev(), generator=torch.Generator(device=dev()).manual_seed(k))
    out = torch.full((m, n), float("nan"), device=dev())
    tb.gguf(m, n, k, name, x_dtype="float32").launch(x, wd, out)
    want = x.double() @ tb.dequantize(wd, name, n, k).double().t()
    # fp32 additions of 8 scale groups (16 for Q6_K) and of 16 slices, each about 2.4e-8 of the running sum: 2.4e-8
    # sqrt(8 / 2 + 16 / 2) = 8e-8, and what an MMA truncates below that; Q4_K has two chains of eight MMAs a slice, which
    # truncate 1.3e-8 each at most
    assert float((out.double() - want).norm() / want.norm()) < (2.6e-7 if name == "q4_k" else 1.3e-7)


@pytest.mark.parametrize("x", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("name,m,k", [("q8_0", 5, 512), ("q4_0", 5, 512), ("q6_k", 5, 512), ("q4_k", 5, 4096), ("q4_k", 12, 4608)])
def test_gemv_frag_special_values(name, m, k, x):
    """Rows with an infinity or a NaN stay with themselves and are what the decoded weights make of them; zero and tiny
    rows keep their scale."""
    n = 2200 if m > 8 else 40
    wd = to_dev(oracle.make_weights(name, n, k, seed=5))
    dtype = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}[x]
    xd = torch.randn(m, k, device=dev(), generator=torch.Generator(device=dev()).manual_seed(1))
    xd[0] = 0
    xd[1] *= 2.0 ** (-14 if x == "f16" else -100)
    xd[2, 7] = float("nan")
    xd[3, 9] = float("inf")
    xd[m - 1, 300] = float("-inf")
    if m > 8:
        xd[7, 4500], xd[7, 4501] = float("inf"), float("inf")
    xd = xd.to(dtype)
    assert tb.ops.gemv_on_registers(name, m, n, k, dtype)
    out = torch.empty((m, n), device=dev())
    tb.gguf(m, n, k, name, x_dtype=dtype).launch(xd, wd, out)
    weight = tb.dequantize(wd, name, n, k).double()
    want = xd.double() @ weight.t()
    assert torch.all(out[0] == 0) and torch.isnan(out[2]).all()
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isfinite(out), finite)
    assert torch.equal(torch.where(torch.isinf(out), out.sign(), 0 * out.nan_to_num()).double(),
                       torch.where(torch.isinf(want), want.sign(), 0 * want.nan_to_num()))
    for row in range(m):
        if finite[row].all() and row:
            assert float((out[row].double() - want[row]).norm() / want[row].norm()) < (2e-5 if name == "q4_k" else 1e-5)


@pytest.mark.parametrize("name,k", [("q6_k", 768), ("q8_0", 4128), ("q4_0", 992), ("q4_k", 4096)])
@pytest.mark.parametrize("n1,n2", [(48, 33), (16, 1), (40, 24)])
def test_gemv_frag_two_weights(name, k, n1, n2):
    """A grouped launch (first weight of whole tiles) and the two launches it stands for agree."""
    m = 6
    x = to_dev(oracle.make_activations(m, k, seed=1, dtype="bf16"), torch.bfloat16)
    ws = [to_dev(oracle.make_weights(name, n, k, seed=n)) for n in (n1, n2)]
    out = torch.full((m, n1 + n2), float("nan"), device=dev())
    tb.ops.gemv_pair(x, ws[0], n1, ws[1], n2, name, k, out=out)
    want = x.double() @ torch.cat([tb.dequantize(w, name, n, k) for w, n in zip(ws, (n1, n2))]).double().t()
    assert float((out.double() - want).norm() / want.norm()) < 1e-5  # exact operands, fp32 sums: a few sqrt(K) 2^-24
    parts = [torch.empty((m, n), device=dev()) for n in (n1, n2)]
    for w, n, part in zip(ws, (n1, n2), parts):
        tb.gemv(x, w, name, n, k, out=part)
    assert float((out - torch.cat(parts, 1)).norm() / out.norm()) < 1e-5
