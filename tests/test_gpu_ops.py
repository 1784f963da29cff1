"""Numerics of every CUDA kernel against the fp32 PyTorch references."""
import math

import pytest
import torch

from omni_npu_b200 import ops
from omni_npu_b200.ops import ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(a, b, atol, rtol):
    torch.testing.assert_close(a.float().cpu(), b.float().cpu(), atol=atol, rtol=rtol)


@pytest.fixture(autouse=True)
def _status():
    yield
    ops.check_status()


# ------------------------------------------------------------------- GEMM
@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (128, 256, 128), (256, 512, 4096), (77, 200, 136),
                                   (1, 4096, 4096), (128, 6144, 4096), (1000, 1024, 2048),
                                   (8192, 4096, 4096)])
def test_gemm_bf16(m, n, k):
    torch.manual_seed(0)
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(n, k, device=DEV, dtype=torch.bfloat16) * 0.05
    out = ops.gemm(a, w)
    want = ref.gemm(a.cpu(), w.cpu())
    _close(out, want, atol=2e-2 * math.sqrt(k / 64), rtol=2e-2)


@pytest.mark.parametrize("bn,splits", [(32, 1), (64, 2), (112, 4), (128, 3), (208, 1), (256, 1), (256, 8),
                                       (64, -2), (112, -4), (128, 8), (96, 5), (16, 7)])
def test_gemm_tile_widths_and_split_k(bn, splits):
    torch.manual_seed(1)
    m, n, k = 200, 1000, 4096
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(n, k, device=DEV, dtype=torch.bfloat16) * 0.05
    out = ops.gemm(a, w, bn=bn, splits=splits)
    _close(out, ref.gemm(a.cpu(), w.cpu()), atol=0.15, rtol=2e-2)
    # split-K leaves its counters at rest: a second call must agree
    out2 = ops.gemm(a, w, bn=bn, splits=splits)
    assert torch.equal(out, out2)


@pytest.mark.parametrize("m,n,k", [(128, 4096, 4096), (64, 6144, 4096), (1, 4096, 14336), (100, 1000, 4104)])
def test_gemm_small_m_default_plan(m, n, k):
    """Decode-shaped problems take the cluster split-K path by default."""
    torch.manual_seed(5)
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(n, k, device=DEV, dtype=torch.bfloat16) * 0.05
    bias = torch.randn(n, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(m, n, device=DEV, dtype=torch.bfloat16)
    out = ops.gemm(a, w, bias, res)
    _close(out, ref.gemm(a.cpu(), w.cpu(), bias.cpu(), res.cpu()), 0.2, 2e-2)
    assert torch.equal(out, ops.gemm(a, w, bias, res))


def test_gemm_epilogues():
    torch.manual_seed(2)
    m, n, k = 300, 768, 1024
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(n, k, device=DEV, dtype=torch.bfloat16) * 0.05
    bias = torch.randn(n, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(m, n, device=DEV, dtype=torch.bfloat16)
    _close(ops.gemm(a, w, bias, res), ref.gemm(a.cpu(), w.cpu(), bias.cpu(), res.cpu()), 0.08, 2e-2)
    _close(ops.gemm(a, w, bias, res, splits=2, bn=128), ref.gemm(a.cpu(), w.cpu(), bias.cpu(), res.cpu()), 0.08, 2e-2)
    _close(ops.gemm(a, w, bias, res, splits=-2), ref.gemm(a.cpu(), w.cpu(), bias.cpu(), res.cpu()), 0.08, 2e-2)
    o32 = ops.gemm(a, w, out_dtype=torch.float32)
    assert o32.dtype == torch.float32
    _close(o32, ref.gemm(a.cpu(), w.cpu(), out_dtype=torch.float32), 2e-2, 1e-2)
    # fused SwiGLU with interleaved gate/up rows
    i = n // 2
    wi = ref.interleave_gate_up(w[:i], w[i:])
    fused = ops.gemm(a, wi, swiglu=True)
    want = ref.silu_and_mul(ref.gemm(a.cpu(), w.cpu(), out_dtype=torch.float32))
    _close(fused, want, 0.06, 3e-2)


@pytest.mark.parametrize("m,n,k,bn", [(256, 256, 128, 0), (512, 1024, 4096, 0), (300, 200, 136, 0),
                                      (1000, 1024, 2048, 128), (8192, 4096, 4096, 0), (257, 96, 64, 96),
                                      (2048, 6144, 4096, 192), (130, 4096, 512, 32)])
def test_gemm_cta_pair(m, n, k, bn):
    """256-row tiles computed by two SMs (tcgen05 cta_group::2)."""
    torch.manual_seed(6)
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(n, k, device=DEV, dtype=torch.bfloat16) * 0.05
    out = ops.gemm(a, w, bn=bn, pair=True)
    torch.cuda.synchronize()
    ops.check_status()
    _close(out, ref.gemm(a.cpu(), w.cpu()), atol=2e-2 * math.sqrt(k / 64), rtol=2e-2)
    assert torch.equal(out, ops.gemm(a, w, bn=bn, pair=True))


def test_gemm_cta_pair_epilogues_and_fp8():
    torch.manual_seed(7)
    m, n, k = 700, 768, 1024
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(n, k, device=DEV, dtype=torch.bfloat16) * 0.05
    bias = torch.randn(n, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(m, n, device=DEV, dtype=torch.bfloat16)
    _close(ops.gemm(a, w, bias, res, pair=True), ref.gemm(a.cpu(), w.cpu(), bias.cpu(), res.cpu()), 0.08, 2e-2)
    o32 = ops.gemm(a, w, out_dtype=torch.float32, pair=True)
    assert o32.dtype == torch.float32
    _close(o32, ref.gemm(a.cpu(), w.cpu(), out_dtype=torch.float32), 2e-2, 1e-2)
    i = n // 2
    wi = ref.interleave_gate_up(w[:i], w[i:])
    fused = ops.gemm(a, wi, swiglu=True, pair=True)
    _close(fused, ref.silu_and_mul(ref.gemm(a.cpu(), w.cpu(), out_dtype=torch.float32)), 0.06, 3e-2)
    a8 = (torch.randn(512, 1024, device=DEV) * 0.5).to(torch.float8_e4m3fn)
    w8 = (torch.randn(512, 1024, device=DEV) * 0.5).to(torch.float8_e4m3fn)
    _close(ops.gemm(a8, w8, pair=True), ref.gemm(a8.cpu(), w8.cpu()), 0.25, 2e-2)
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("m,n,k", [(128, 256, 256), (200, 1000, 4096), (1, 4096, 4096), (777, 6144, 1024)])
def test_gemm_int8_scaled(m, n, k):
    """int8 x int8 with s32 accumulation on the tensor cores; per-token x per-channel scales."""
    torch.manual_seed(8)
    x = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(n, k, device=DEV) * 0.05
    xq, xs = ops.quant_int8_per_token(x)
    rq, rs = ref.quant_int8_per_token(x.cpu())
    assert (xq.cpu().int() - rq.int()).abs().max() <= 1 and torch.allclose(xs.cpu(), rs, rtol=1e-3)
    ws = w.abs().amax(dim=1) / 127.0
    wq = torch.round(w / ws[:, None]).clamp(-127, 127).to(torch.int8)
    bias = torch.randn(n, device=DEV, dtype=torch.bfloat16)
    out = ops.gemm_scaled(xq, wq, xs, ws, bias, out_dtype=torch.float32)
    torch.cuda.synchronize()
    ops.check_status()
    want = ref.gemm_scaled(xq.cpu(), wq.cpu(), xs.cpu(), ws.cpu(), bias.cpu(), out_dtype=torch.float32)
    _close(out, want, atol=2e-3 * math.sqrt(k / 64), rtol=1e-3)     # integer accumulation is exact
    # against the unquantised product: quantisation error only
    full = x.float().cpu() @ w.cpu().t() + bias.float().cpu()
    assert (out.cpu() - full).abs().max() < 0.05 * full.abs().max() + 0.05


def test_gemm_fp8_scaled():
    torch.manual_seed(9)
    m, n, k = 300, 512, 1024
    a = (torch.randn(m, k, device=DEV) * 0.5).to(torch.float8_e4m3fn)
    w = (torch.randn(n, k, device=DEV) * 0.5).to(torch.float8_e4m3fn)
    sa = torch.rand(m, device=DEV) + 0.5
    sw = torch.rand(n, device=DEV) + 0.5
    out = ops.gemm_scaled(a, w, sa, sw, out_dtype=torch.float32)
    want = (a.float().cpu() @ w.float().cpu().t()) * sa.cpu()[:, None] * sw.cpu()[None, :]
    _close(out, want, atol=0.05, rtol=1e-2)


def test_grouped_gemm():
    torch.manual_seed(3)
    e, n, k = 8, 512, 1024
    counts = [0, 5, 128, 129, 300, 1, 0, 77]
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32)
    rows = int(offs[-1])
    a = torch.randn(rows, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(e, n, k, device=DEV, dtype=torch.bfloat16) * 0.05
    out = ops.grouped_gemm(a, w, offs.to(DEV))
    _close(out, ref.grouped_gemm(a.cpu(), w.cpu(), offs), 0.08, 2e-2)
    wi = ref.interleave_gate_up(w[:, : n // 2], w[:, n // 2:])
    out = ops.grouped_gemm(a, wi, offs.to(DEV), swiglu=True)
    want = ref.silu_and_mul(ref.grouped_gemm(a.cpu().float(), w.cpu().float(), offs))
    _close(out, want, 0.06, 3e-2)


@pytest.mark.parametrize("m,n,k", [(1, 128, 64), (1, 6144, 4096), (15, 1000, 520), (16, 4096, 14336), (17, 24, 2048),
                                   (33, 28672, 256), (63, 40000, 128), (5, 130, 8), (128, 20000, 64), (100, 18945, 72)])
def test_gemm_few_rows(m, n, k):
    """Weights as the M operand: every tile width, K splits of 1 to 8, ragged N and K, all epilogues."""
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = (torch.randn(n, k, device=DEV) * k ** -0.5).bfloat16()
    bias = torch.randn(n, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(m, n, device=DEV, dtype=torch.bfloat16)
    exact = a.double() @ w.double().T
    # fp32 sums of k products of size k ** -0.5: k * 2 ** -24 of their absolute sum at worst
    _close(ops.gemm(a, w, out_dtype=torch.float32), exact.float(), k ** 0.5 * 2 ** -22 + 1e-6, 0)
    # one rounding to bf16
    _close(ops.gemm(a, w, bias, res), (exact + bias.double() + res.double()).float(), 1e-3, 2 ** -8)
    _close(ops.gemm(a, w, bias, unary="relu2"), (exact.clamp_min(0) ** 2 + bias.double()).float(), 1e-3, 2 ** -8)
    if n % 16 == 0:
        gate, up = exact.view(m, -1, 2, 8).unbind(2)
        _close(ops.gemm(a, w, swiglu=True), (torch.nn.functional.silu(gate) * up).reshape(m, -1).float(), 1e-3, 2 ** -7)
    # a row's result does not depend on the rows beside it
    assert torch.equal(ops.gemm(a[:1], w), ops.gemm(a, w)[:1])
    ops.check_status()


@pytest.mark.parametrize("m,n,k", [(63, 2048, 576), (64, 130, 576), (33, 1000, 1024), (3, 48, 4096), (62, 258, 2048), (128, 56, 4096)])
def test_gemm_few_rows_split(m, n, k):
    """Sums over the CTAs of a cluster, four columns at a time: columns left over, results and residuals off 16 bytes."""
    torch.manual_seed(m + n + k)
    assert ops._core().gemm_stream_splits(n, k, 0, 148) > 1
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = (torch.randn(n, k, device=DEV) * k ** -0.5).bfloat16()
    bias = torch.randn(n, device=DEV, dtype=torch.bfloat16)
    exact = a.double() @ w.double().T
    _close(ops.gemm(a, w, out_dtype=torch.float32), exact.float(), k ** 0.5 * 2 ** -22 + 1e-6, 0)
    # one rounding to bf16
    _close(ops.gemm(a, w, bias, unary="relu2"), (exact.clamp_min(0) ** 2 + bias.double()).float(), 1e-3, 2 ** -8)
    for shift in (0, 1, 2):
        res = torch.randn(m * n + 4, device=DEV, dtype=torch.bfloat16)[shift: shift + m * n].view(m, n)
        _close(ops.gemm(a, w, bias, res), (exact + bias.double() + res.double()).float(), 1e-3, 2 ** -8)
    if n % 16 == 0:
        gate, up = (exact + bias.double()).view(m, -1, 2, 8).unbind(2)
        _close(ops.gemm(a, w, bias, swiglu=True), (torch.nn.functional.silu(gate) * up).reshape(m, -1).float(), 1e-3, 2 ** -7)


@pytest.mark.parametrize("n,k", [(64, 2048), (256, 7168), (4096, 4096), (6144, 4096), (9216, 2048), (12288, 2048), (18944, 1024),
                                 (20000, 512), (2048, 512), (5632, 2048), (1000, 1408), (48, 256), (130, 4096)])
def test_a_row_does_not_depend_on_the_rows_beside_it(n, k, monkeypatch):
    """1 to 128 rows, on whichever kernels: a decode step padded to a captured size gives the unpadded one's numbers.
    (Plain products of 64 rows and more may be cuBLAS's.)"""
    torch.manual_seed(n + k)
    a = torch.randn(128, k, device=DEV, dtype=torch.bfloat16)
    w = (torch.randn(n, k, device=DEV) * k ** -0.5).bfloat16()
    res = torch.randn(128, n, device=DEV, dtype=torch.bfloat16)
    forms = [lambda m: ops.gemm(a[:m], w, out_dtype=torch.float32), lambda m: ops.gemm(a[:m], w, residual=res[:m]),
             lambda m: ops.gemm(a[:m], w, unary="relu2")] + ([lambda m: ops.gemm(a[:m], w, swiglu=True)] if n % 16 == 0 else [])
    monkeypatch.setattr(ops, "SMALL_M_GEMM", "own")
    forms.append(lambda m: ops.gemm(a[:m], w))
    for form in forms:
        want = form(128)
        for m in (1, 15, 16, 17, 33, 63, 64, 65, 96, 127):
            assert torch.equal(form(m), want[:m]), (m,)


@pytest.mark.parametrize("n,k", [(4096, 2048), (640, 1024), (18432, 512), (130, 256)])
def test_an_e4m3_row_does_not_depend_on_the_rows_beside_it(n, k):
    """On either side of the 64 rows that the weight-streaming kernel takes."""
    torch.manual_seed(n + k)
    q, s = ops.quant_fp8_1x128(torch.randn(300, k, device=DEV, dtype=torch.bfloat16))
    w, ws = torch.randn(n, k, device=DEV).to(torch.float8_e4m3fn), torch.rand(-(-n // 128), k // 128, device=DEV)
    want = ops.gemm_fp8_block(q, s, w, ws, out_dtype=torch.float32)
    few = ops.gemm_fp8_block(q[:64], s[:64], w, ws, out_dtype=torch.float32)
    for m in (1, 31, 32, 33, 63):
        assert torch.equal(ops.gemm_fp8_block(q[:m], s[:m], w, ws, out_dtype=torch.float32), few[:m]), (m,)
    for m in (65, 128, 129, 257):
        assert torch.equal(ops.gemm_fp8_block(q[:m], s[:m], w, ws, out_dtype=torch.float32), want[:m]), (m,)


@pytest.mark.parametrize("m,n,k", [(65, 18944, 72), (129, 20000, 200), (257, 130, 64), (300, 1000, 136), (1023, 384, 1048),
                                   (1025, 257, 8), (2000, 48, 520), (33, 304, 128)])
def test_gemm_pair_rows(m, n, k):
    """Rows of A as the N operand of CTA pairs: every width of a tile, ragged M, N and K, all epilogues."""
    torch.manual_seed(m + n)
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = (torch.randn(n, k, device=DEV) * k ** -0.5).bfloat16()
    bias = torch.randn(n, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(m, n, device=DEV, dtype=torch.bfloat16)
    exact = a.double() @ w.double().T
    for bn in (0, 32, 160, 224, 256):
        _close(ops.gemm(a, w, bn=bn, pair=True), exact.float(), 1e-3, 2 ** -8)
    # fp32 sums of k products of size k ** -0.5; else one rounding to bf16
    _close(ops.gemm(a, w, out_dtype=torch.float32, pair=True), exact.float(), k ** 0.5 * 2 ** -22 + 1e-6, 0)
    _close(ops.gemm(a, w, bias, res, pair=True), (exact + bias.double() + res.double()).float(), 1e-3, 2 ** -8)
    _close(ops.gemm(a, w, bias, unary="relu2", pair=True), (exact.clamp_min(0) ** 2 + bias.double()).float(), 1e-3, 2 ** -8)
    if n % 16 == 0:
        gate, up = (exact + bias.double()).view(m, -1, 2, 8).unbind(2)
        _close(ops.gemm(a, w, bias, swiglu=True), (torch.nn.functional.silu(gate) * up).reshape(m, -1).float(), 1e-3, 2 ** -7)
    ops.check_status()


@pytest.mark.parametrize("counts,n,k", [
    ([1], 128, 64), ([0, 16, 17, 0, 1, 200, 0], 256, 320), ([64, 65, 0, 63], 1000, 96), ([0, 0, 0, 3], 48, 40),
    ([1] * 70, 144, 128), ([300] + [0] * 11, 384, 256), ([255, 256, 257, 0, 31, 33, 513], 304, 136), ([2049], 2048, 8),
    ([2600, 3], 512, 200), ([900, 100], 100, 64), ([129] * 70, 135, 72), ([33] * 200, 264, 64)])
def test_grouped_gemm_tiles(counts, n, k):
    """The weight-streaming kernel and the one on CTA pairs: ragged rows, rows of a tile dealt out evenly, odd N."""
    torch.manual_seed(len(counts) + n)
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32)
    rows, e = int(offs[-1]), len(counts)
    a = torch.randn(rows + 5, k, device=DEV, dtype=torch.bfloat16)      # rows past the last offset take no part
    w = (torch.randn(e, n, k, device=DEV) * k ** -0.5).bfloat16()
    exact = torch.cat([a[offs[i]: offs[i + 1]].double() @ w[i].double().T for i in range(e)])
    # one rounding to bf16 (2 ** -9 relative), and of two products of fp32 activations
    _close(ops.grouped_gemm(a, w, offs.to(DEV))[:rows], exact.float(), 1e-3, 2 ** -8)
    _close(ops.grouped_gemm(a, w, offs.to(DEV), unary="relu2")[:rows], (exact.clamp_min(0) ** 2).float(), 1e-3, 2 ** -8)
    if n % 16 == 0:
        gate, up = exact.view(rows, -1, 2, 8).unbind(2)
        _close(ops.grouped_gemm(a, w, offs.to(DEV), swiglu=True)[:rows],
               (torch.nn.functional.silu(gate) * up).reshape(rows, -1).float(), 1e-3, 2 ** -7)
    ops.check_status()


@pytest.mark.parametrize("m,n,k", [(5, 256, 4096), (128, 20480, 1024), (300, 20480, 1024), (100, 4096, 4096), (1100, 2048, 1024)])
def test_products_wait_for_weights_written_right_ahead(m, n, k):
    """An operand that the kernel ahead writes, in memory that held another one: read once that kernel is through."""
    torch.manual_seed(m)
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    q, s = ops.quant_fp8_1x128(a)
    res = torch.randn(m, n, device=DEV, dtype=torch.bfloat16)
    ones, scale = torch.ones(k, device=DEV, dtype=torch.bfloat16), torch.rand(-(-n // 128), k // 128, device=DEV)
    row, col = torch.rand(m, device=DEV), torch.rand(n, device=DEV)
    sources = [torch.randn(n, k, device=DEV, dtype=torch.bfloat16) for _ in range(4)]
    calls = [(lambda x: ops.rms_norm(x, ones, 1e-6), lambda w: ops.gemm(a, w)),
             (lambda x: ops.rms_norm(x, ones, 1e-6), lambda w: ops.gemm(a, w, residual=res)),
             (lambda x: ops.quant_fp8_1x128(x)[0], lambda w: ops.gemm_fp8_block(q, s, w, scale)),
             (lambda x: ops.quant_fp8_1x128(x)[0], lambda w: ops.gemm_scaled(q, w, row, col))]
    for write, product in calls:
        for i in range(12):
            w = write(sources[i % 4])
            got = product(w)
            torch.cuda.synchronize()
            assert torch.equal(got, product(w))
            del w, got
    h = torch.randn(64, 8192, device=DEV, dtype=torch.bfloat16)
    batched = torch.randn(3, 16, 128, device=DEV, dtype=torch.bfloat16)
    for i in range(12):
        w = ops.rms_norm(sources[i % 4].view(-1, 1024)[:1024], ones[:1024], 1e-6).view(16, 512, 128)
        got = ops.batched_gemm(batched, w, h.new_empty(3, 16, 512))
        torch.cuda.synchronize()
        assert torch.equal(got, ops.batched_gemm(batched, w, h.new_empty(3, 16, 512)))
        del w, got


@pytest.mark.parametrize("rows,h", [(5999, 1024), (6000, 1024), (6001, 1280), (6000, 1288), (7000, 1016)])
def test_norm_of_many_short_rows(rows, h):
    """On either side of the sizes at which a row takes a warp and a CTA."""
    torch.manual_seed(rows)
    x, w = torch.randn(rows, h, device=DEV).bfloat16(), (torch.rand(h, device=DEV) + 0.5).bfloat16()
    want = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    _close(ops.rms_norm(x, w, 1e-6), want.float(), 1e-3, 2 ** -8)      # one rounding to bf16


@pytest.mark.parametrize("rows,h", [(1, 1024), (40, 4096), (3, 16384)])
def test_norm_waits_for_weights_written_right_ahead(rows, h):
    torch.manual_seed(h)
    x, ones = torch.randn(rows, h, device=DEV, dtype=torch.bfloat16), torch.ones(h, device=DEV, dtype=torch.bfloat16)
    sources = [torch.randn(1, h, device=DEV, dtype=torch.bfloat16) for _ in range(4)]
    for i in range(24):
        w = ops.rms_norm(sources[i % 4], ones, 1e-6)[0]
        got, res = ops.rms_norm(x, w, 1e-6), x.clone()
        added = ops.fused_add_rms_norm(x, res, ops.rms_norm(sources[(i + 1) % 4], ones, 1e-6)[0], 1e-6)
        torch.cuda.synchronize()
        exact = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-6)
        # one rounding to bf16; of the doubled row nothing changes but the weight of eps
        _close(got, (exact * w.double()).float(), 1e-3, 2 ** -8)
        other = ops.rms_norm(sources[(i + 1) % 4], ones, 1e-6)[0]
        _close(added, (exact * other.double()).float(), 1e-3, 2 ** -8)
        del w, got, added, other


@pytest.mark.parametrize("counts,n,k", [([17] * 8, 128, 1024), ([0, 70, 3, 128], 48, 2048), ([300] * 3, 128, 776), ([33, 0, 20], 16, 4096)])
def test_grouped_gemm_narrow(counts, n, k):
    """A single tile of weight rows per group and a long K, into rows of a wider tensor too."""
    torch.manual_seed(n + k)
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32)
    rows, e = int(offs[-1]), len(counts)
    assert ops.grouped_rows_tile(rows, e, n, k) == -1
    a = torch.randn(rows, k, device=DEV, dtype=torch.bfloat16)
    w = (torch.randn(e, n, k, device=DEV) * k ** -0.5).bfloat16()
    exact = torch.cat([a[offs[i]: offs[i + 1]].double() @ w[i].double().T for i in range(e)])
    out = torch.zeros(rows, 256, device=DEV, dtype=torch.bfloat16)
    # one rounding to bf16
    _close(ops.grouped_gemm(a, w, offs.to(DEV), out=out[:, :n]), exact.float(), 1e-3, 2 ** -8)
    assert not out[:, n:].any()
    gate, up = exact.view(rows, -1, 2, 8).unbind(2)
    _close(ops.grouped_gemm(a, w, offs.to(DEV), swiglu=True), (torch.nn.functional.silu(gate) * up).reshape(rows, -1).float(),
           1e-3, 2 ** -7)
    ops.check_status()


def test_gemm_fp8_plain():
    torch.manual_seed(4)
    m, n, k = 256, 512, 1024
    a = (torch.randn(m, k, device=DEV) * 0.5).to(torch.float8_e4m3fn)
    w = (torch.randn(n, k, device=DEV) * 0.5).to(torch.float8_e4m3fn)
    out = ops.gemm(a, w)
    _close(out, ref.gemm(a.cpu(), w.cpu()), 0.25, 2e-2)


# --------------------------------------------------------------- row kernels
@pytest.mark.parametrize("t,h", [(1, 4096), (37, 4096), (128, 2048), (5, 7168), (16, 128), (33, 16384)])
def test_rms_norm(t, h):
    torch.manual_seed(0)
    x = torch.randn(t, h, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(h, device=DEV, dtype=torch.bfloat16)
    _close(ops.rms_norm(x, w, 1e-6), ref.rms_norm(x.cpu(), w.cpu(), 1e-6), 2e-2, 2e-2)
    r = torch.randn(t, h, device=DEV, dtype=torch.bfloat16)
    r_ref = r.cpu().clone()
    y = ops.fused_add_rms_norm(x, r, w, 1e-6)
    y_ref = ref.fused_add_rms_norm(x.cpu(), r_ref, w.cpu(), 1e-6)
    _close(r, r_ref, 1e-2, 1e-2)
    _close(y, y_ref, 3e-2, 2e-2)


def test_rms_norm_strided_heads():
    x = torch.randn(9, 3 * 128 * 4, device=DEV, dtype=torch.bfloat16)
    q = x[:, : 128 * 4]
    w = torch.randn(128, device=DEV, dtype=torch.bfloat16)
    got = ops.rms_norm(q.reshape(-1, 128), w, 1e-6)
    _close(got, ref.rms_norm(q.cpu().reshape(-1, 128), w.cpu(), 1e-6), 2e-2, 2e-2)


def test_silu_and_mul_and_quant():
    x = torch.randn(50, 2 * 1408, device=DEV, dtype=torch.bfloat16)
    _close(ops.silu_and_mul(x), ref.silu_and_mul(x.cpu()), 2e-2, 2e-2)
    y = torch.randn(19, 1024, device=DEV, dtype=torch.bfloat16) * 3
    q, s = ops.quant_fp8_1x128(y)
    qr, sr = ref.quant_fp8_1x128(y.cpu())
    _close(s, sr, 1e-6, 1e-5)
    deq = q.float().view(19, 8, 128) * s.unsqueeze(-1)
    _close(deq.view(19, 1024), y, 0.25, 0.07)


@pytest.mark.parametrize("neox", [True, False])
@pytest.mark.parametrize("rot", [128, 64])
def test_rope_qk(neox, rot):
    t, hq, hk, d = 23, 8, 2, 128
    q = torch.randn(t, hq * d, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(t, hk * d, device=DEV, dtype=torch.bfloat16)
    pos = torch.randint(0, 4000, (t,), device=DEV, dtype=torch.int32)
    cs = ref.build_cos_sin_cache(rot, 4096, 10000.0).to(DEV)
    qr, kr = ref.rope_qk(q.cpu(), k.cpu(), pos.cpu(), cs.cpu(), d, rot, neox)
    ops.rope_qk_(q, k, pos, cs, d, rot, neox)
    _close(q, qr, 2e-2, 2e-2)
    _close(k, kr, 2e-2, 2e-2)


@pytest.mark.parametrize("interleaved", [False, True])
def test_mrope(interleaved):
    t, hq, hk, d = 11, 4, 2, 128
    q = torch.randn(t, hq * d, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(t, hk * d, device=DEV, dtype=torch.bfloat16)
    pos = torch.randint(0, 500, (3, t), device=DEV, dtype=torch.int32)
    cs = ref.build_cos_sin_cache(d, 512, 10000.0).to(DEV)
    sec = (24, 20, 20)
    qr, kr = ref.rope_qk(q.cpu(), k.cpu(), pos.cpu(), cs.cpu(), d, d, True, sec, interleaved)
    ops.rope_qk_(q, k, pos, cs, d, d, True, sec, interleaved)
    _close(q, qr, 2e-2, 2e-2)
    _close(k, kr, 2e-2, 2e-2)


def _paged_setup(seq_lens, q_lens, hq, hk, d, bs, dv=None, seed=0):
    torch.manual_seed(seed)
    dv = dv or d
    b = len(seq_lens)
    max_blocks = max((s + bs - 1) // bs for s in seq_lens) + 1
    nblocks = b * max_blocks + 3
    perm = torch.randperm(nblocks)[: b * max_blocks].view(b, max_blocks).to(torch.int32)
    k_cache = torch.randn(nblocks, hk, bs, d, dtype=torch.bfloat16)
    v_cache = torch.randn(nblocks, hk, bs, dv, dtype=torch.bfloat16)
    t = sum(q_lens)
    q = torch.randn(t, hq * d, dtype=torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    sl = torch.tensor(seq_lens, dtype=torch.int32)
    return q, k_cache, v_cache, perm, cu, sl


@pytest.mark.parametrize("tc", [True, False])
@pytest.mark.parametrize("seq_lens,q_lens,hq,hk,bs,causal", [
    ([130, 64, 517, 9], [130, 33, 200, 9], 8, 2, 16, True),        # with cached context, ragged tiles
    ([1000, 1], [1000, 1], 4, 4, 16, True),                        # many key tiles, a one-row sequence
    ([300, 257], [300, 129], 16, 2, 32, True),                     # 8 query heads per kv head, 32-token blocks
    ([200, 77], [200, 40], 8, 2, 16, False),                       # not causal
    ([640], [64], 8, 1, 64, True),                                 # short chunk over a long context, 64-token blocks
])
def test_gqa_prefill_tcgen05_matches_reference(seq_lens, q_lens, hq, hk, bs, causal, tc):
    """Head size 128: the tcgen05 / TMEM kernel and the mma.sync kernel against the fp32 reference."""
    d = 128
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, q_lens, hq, hk, d, bs, seed=31)
    want, lse_want = ref.paged_attention(q, kc, vc, bt, cu, sl, hq, d ** -0.5, causal, 0, True)
    got, lse = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV),
                               len(seq_lens), max(q_lens), hq, d ** -0.5, causal, 0, True, tcgen05=tc)
    _close(got, want, 2e-2, 2e-2)
    _close(lse, lse_want, 2e-2, 1e-2)
    # q as a column slice of a wider activation (the fused qkv projection's output)
    wide = torch.randn(q.shape[0], q.shape[1] + 512, dtype=torch.bfloat16)
    wide[:, : q.shape[1]] = q
    got2 = ops.gqa_prefill(wide.to(DEV)[:, : q.shape[1]], kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV),
                           sl.to(DEV), len(seq_lens), max(q_lens), hq, d ** -0.5, causal, tcgen05=tc)
    _close(got2, want, 2e-2, 2e-2)


@pytest.mark.parametrize("d,hq,hk,bs,seq_lens,q_lens", [
    (128, 8, 2, 16, [129, 128, 127, 257], [129, 128, 1, 256]),      # heads in pairs: edges of the 128-row / -key tiles
    (128, 6, 2, 16, [257, 255, 400], [257, 129, 128]),              # three heads per key head: row tiles in pairs
    (192, 4, 4, 16, [256, 385, 130], [256, 300, 2]),                # latent prompt sizes, one head per key head
    (192, 4, 2, 64, [140], [140]),
    (128, 4, 1, 128, [300], [300]),                                 # copies of 128 rows
    (128, 32, 4, 8, [700, 1, 650, 90, 513], [700, 1, 600, 5, 513]),  # more items than SMs, smallest copies
])
@pytest.mark.parametrize("causal", [True, False])
def test_gqa_prefill_two_tiles(d, hq, hk, bs, seq_lens, q_lens, causal):
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, q_lens, hq, hk, d, bs, dv=128, seed=3)
    q[: q_lens[0]] *= 4.0                      # scores far apart: the reference maximum moves
    want, lse_want = ref.paged_attention(q, kc, vc, bt, cu, sl, hq, d ** -0.5, causal, 0, True)
    for _ in range(2):
        got, lse = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV),
                                   len(seq_lens), max(q_lens), hq, d ** -0.5, causal, 0, True)
        # P and the result are rounded to bf16 (2^-9 each) of values up to about 4
        _close(got, want, 2e-2, 2e-2)
        _close(lse, lse_want, 2e-2, 1e-2)


@pytest.mark.parametrize("d,hq,hk", [(128, 8, 2), (128, 64, 8), (192, 4, 2)])
@pytest.mark.parametrize("seq_lens,q_lens", [([17], [17]), ([128, 1], [128, 1]), ([64, 65], [64, 65]), ([192, 193, 63], [128, 100, 1]),
                                             ([129, 5], [129, 5])])
@pytest.mark.parametrize("causal", [True, False])
def test_gqa_prefill_small(d, hq, hk, seq_lens, q_lens, causal):
    """Few short prompts, a query tile per CTA, and key tiles of which only the first half exists."""
    test_gqa_prefill_two_tiles(d, hq, hk, 16, seq_lens, q_lens, causal)


@pytest.mark.parametrize("d,bs", [(128, 16), (64, 16), (128, 128)])
def test_gqa_prefill(d, bs):
    seq_lens, q_lens = [130, 64, 517, 9], [130, 33, 200, 9]
    hq, hk = 8, 2
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, q_lens, hq, hk, d, bs)
    want, lse_want = ref.paged_attention(q, kc, vc, bt, cu, sl, hq, d ** -0.5, True, 0, True)
    got, lse = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV),
                               len(seq_lens), max(q_lens), hq, d ** -0.5, True, 0, True)
    _close(got, want, 2e-2, 2e-2)
    _close(lse, lse_want, 2e-2, 1e-2)


def test_gqa_prefill_window_and_mla_dims():
    seq_lens, q_lens = [300, 77], [300, 40]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, q_lens, 4, 4, 128, 16, seed=5)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 4, 0.1, True, 64)
    got = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV), 2, 300,
                          4, 0.1, True, 64)
    _close(got, want, 2e-2, 2e-2)
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, q_lens, 4, 4, 192, 16, dv=128, seed=6)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 4, 192 ** -0.5, True, 0)
    got = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV), 2, 300,
                          4, 192 ** -0.5, True, 0)
    _close(got, want, 2e-2, 2e-2)


@pytest.mark.parametrize("persistent", [2, True, False])
@pytest.mark.parametrize("splits", [1, 2, 5])
@pytest.mark.parametrize("hq,hk,d", [(32, 8, 128), (4, 2, 64), (16, 1, 128), (16, 2, 128)])
def test_gqa_decode(splits, hq, hk, d, persistent):
    seq_lens = [1, 17, 64, 65, 1000, 333]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [1] * 6, hq, hk, d, 16, seed=7)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, hq, d ** -0.5, True, 0)
    got = ops.gqa_decode(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), 6, hq, d ** -0.5,
                         splits=splits, persistent=persistent)
    _close(got, want, 2e-2, 2e-2)


def test_gqa_decode_persistent_more_items_than_ctas_twice():
    """More (sequence, kv head, split) items than resident CTAs: every CTA walks several items
    handed out by the device counter; the counter is back at zero afterwards, so a second call
    (as a graph replay would make it) gives the same result."""
    torch.manual_seed(21)
    seq_lens = [int(x) for x in torch.randint(1, 700, (96,))]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [1] * 96, 32, 8, 128, 16, seed=22)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 32, 128 ** -0.5, True, 0)
    args = (q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), 96, 32, 128 ** -0.5)
    for splits in (1, 2):
        for _ in range(2):
            got = ops.gqa_decode(*args, splits=splits, persistent=True)
            _close(got, want, 2e-2, 2e-2)
    wc = ops.device_state(torch.device("cuda", 0)).work_counter(torch.cuda.current_stream().cuda_stream)
    assert wc.tolist() == [0, 0]
    assert ops.decode_splits_persistent(128, 8, 1296) == 2 and ops.decode_splits_persistent(128, 4, 1296) == 4
    assert ops.decode_splits_persistent(1, 8, 8192) > 8          # few items: split to fill the SMs


@pytest.mark.parametrize("n_seqs,hq,hk,hi", [(96, 32, 8, 700), (300, 8, 2, 150), (3, 16, 1, 5000), (40, 4, 4, 64)])
def test_gqa_decode_balanced_cut(n_seqs, hq, hk, hi):
    """Persistent CTAs over the balanced cut of the key tiles: ranges that hold several whole items,
    items that spread over many CTAs, more CTAs than tiles; twice, as a graph replay would run it."""
    torch.manual_seed(31)
    seq_lens = [int(x) for x in torch.randint(1, hi, (n_seqs,))]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [1] * n_seqs, hq, hk, 128, 16, seed=32)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, hq, 128 ** -0.5, True, 0)
    args = (q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), n_seqs, hq, 128 ** -0.5)
    for _ in range(2):
        got = ops.gqa_decode(*args, persistent=2)
        _close(got, want, 2e-2, 2e-2)
    ops.check_status()


def test_gqa_decode_balanced_cut_multi_token_window_and_sink():
    seq_lens = [40, 130, 7, 900]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [3] * 4, 8, 2, 128, 16, seed=33)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 8, 0.09, True, 0)
    got = ops.gqa_decode(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), 4, 8, 0.09, q_len=3,
                         persistent=2)
    _close(got, want, 2e-2, 2e-2)
    seq_lens = [1, 17, 64, 65, 1000, 333]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [1] * 6, 8, 2, 128, 16, seed=13)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 8, 0.1, True, 64, False, 32)
    got = ops.gqa_decode(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), 6, 8, 0.1, window=64,
                         sink=32, persistent=2)
    _close(got, want, 2e-2, 2e-2)
    # head size 64, sixteen query rows per kv head
    seq_lens = [500, 3, 129]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [1] * 3, 16, 1, 64, 16, seed=34)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 16, 0.125, True, 0)
    got = ops.gqa_decode(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), 3, 16, 0.125, persistent=2)
    _close(got, want, 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("persistent", [2, 1, 0])
def test_gqa_decode_two_tokens_eight_rows(persistent):
    """Two new tokens per sequence with a group of four: eight query rows per kv head, the
    transposed-product path of the decode kernels, each query with its own causal limit."""
    seq_lens = [40, 130, 7, 64, 2, 700]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [2] * 6, 8, 2, 128, 16, seed=35)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 8, 0.09, True, 0)
    for splits in (1, 3):
        got = ops.gqa_decode(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), 6, 8, 0.09, q_len=2,
                             splits=splits, persistent=persistent)
        _close(got, want, 2e-2, 2e-2)
    ops.check_status()


def test_gqa_decode_multi_token():
    seq_lens = [40, 130, 7]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [3] * 3, 8, 2, 128, 16, seed=8)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 8, 0.09, True, 0)
    got = ops.gqa_decode(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), 3, 8, 0.09, q_len=3,
                         splits=2)
    _close(got, want, 2e-2, 2e-2)


@pytest.mark.parametrize("window,sink", [(64, 32), (16, 16), (200, 48)])
def test_gqa_window_with_sink_tokens(window, sink):
    """Sliding-window attention where the first `sink` cached tokens stay visible."""
    seq_lens, q_lens = [300, 77, 40], [300, 40, 1]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, q_lens, 8, 2, 128, 16, seed=12)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 8, 0.1, True, window, False, sink)
    got = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV), 3, 300,
                          8, 0.1, True, window, sink=sink)
    _close(got, want, 2e-2, 2e-2)
    # without the sink the result differs (the mask matters) ...
    nosink = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV), 3, 300,
                             8, 0.1, True, window)
    assert (nosink.float().cpu() - want.float()).abs().max() > 1e-2
    # ... and decode agrees too
    seq_lens = [1, 17, 64, 65, 1000, 333]
    q, kc, vc, bt, cu, sl = _paged_setup(seq_lens, [1] * 6, 8, 2, 128, 16, seed=13)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, 8, 0.1, True, window, False, sink)
    for splits in (1, 3):
        got = ops.gqa_decode(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), sl.to(DEV), 6, 8, 0.1,
                             window=window, splits=splits, sink=sink)
        _close(got, want, 2e-2, 2e-2)


def test_lse_merge_and_gather_cache():
    torch.manual_seed(14)
    n, t, h, d = 3, 37, 8, 128
    outs = torch.randn(n, t, h, d, device=DEV, dtype=torch.bfloat16)
    lses = torch.randn(n, t, h, device=DEV) * 3
    lses[1, 5] = float("-inf")                      # a partial that saw no key
    lses[:, 9, 2] = float("-inf")                   # nobody saw a key
    got, lse = ops.merge_attn_states(outs, lses)
    want, lse_want = ref.merge_attn_states(outs.cpu(), lses.cpu())
    _close(got, want, 2e-2, 2e-2)
    assert torch.isinf(lse[9, 2]) and float(got[9, 2].abs().sum()) == 0
    fin = ~torch.isinf(lse_want)
    _close(lse.cpu()[fin], lse_want[fin], 1e-3, 1e-3)
    # merging the two halves of a key set reproduces attention over the whole set
    q = torch.randn(4, 64)
    k, v = torch.randn(50, 64), torch.randn(50, 64)
    def part(ks, vs):
        s_ = q @ ks.t()
        l_ = torch.logsumexp(s_, -1)
        return torch.softmax(s_, -1) @ vs, l_
    (o1, l1), (o2, l2) = part(k[:20], v[:20]), part(k[20:], v[20:])
    whole, _ = part(k, v)
    m_out, _ = ops.merge_attn_states(torch.stack([o1, o2]).unsqueeze(2).to(DEV, torch.bfloat16),
                                     torch.stack([l1, l2]).unsqueeze(2).to(DEV))
    _close(m_out[:, 0], whole, 3e-2, 3e-2)
    cache = torch.randn(12, 16, 576, device=DEV, dtype=torch.bfloat16)
    bt = torch.tensor([[3, 7, 1, 0], [11, 2, 0, 0]], dtype=torch.int32, device=DEV)
    sl = torch.tensor([40, 17], dtype=torch.int32)
    assert torch.equal(ops.gather_cache(cache, bt, sl).cpu(), ref.gather_cache(cache.cpu(), bt.cpu(), sl))


@pytest.mark.parametrize("m,n,k", [(1, 4096, 7168), (33, 130, 128), (64, 1000, 640), (17, 7168, 2048), (5, 40000, 256)])
def test_gemm_fp8_few_rows(m, n, k, monkeypatch):
    """The weight-streaming block-scaled kernel against the one that it stands in for: K splits of 1 to 8, ragged N, epilogues."""
    torch.manual_seed(m + n)
    w = torch.randn(n, k, device=DEV).to(torch.float8_e4m3fn)
    ws = torch.rand(-(-n // 128), k // 128, device=DEV) + 0.5
    q, s = ops.quant_fp8_1x128(torch.randn(m, k, device=DEV, dtype=torch.bfloat16))
    bias, res = torch.randn(n, device=DEV).bfloat16(), torch.randn(m, n, device=DEV).bfloat16()
    got = [ops.gemm_fp8_block(q, s, w, ws, **kw) for kw in (dict(out_dtype=torch.float32), dict(bias=bias, residual=res))]
    monkeypatch.setattr(ops, "FP8_STREAM_ROWS", 0)
    want = [ops.gemm_fp8_block(q, s, w, ws, **kw) for kw in (dict(out_dtype=torch.float32), dict(bias=bias, residual=res))]
    # the same fp32 products, summed in another order where K is split; one rounding to bf16
    _close(got[0], want[0], 1e-5 * k ** 0.5, 1e-5)
    _close(got[1], want[1], 1e-2, 2 ** -7)
    ops.check_status()


@pytest.mark.parametrize("counts,n,k,swiglu", [([0, 5, 64, 65, 0, 16, 17, 1], 512, 256, True), ([3], 130, 128, False),
                                               ([33] * 40, 256, 384, True), ([0, 0, 90], 1000, 640, False)])
def test_grouped_gemm_fp8_few_rows(counts, n, k, swiglu, monkeypatch):
    torch.manual_seed(n)
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device=DEV)
    rows, e = sum(counts), len(counts)
    assert rows <= ops.FP8_STREAM_GROUP_ROWS * e
    w = torch.randn(e, n, k, device=DEV).to(torch.float8_e4m3fn)
    up = n // 256 if swiglu else 0
    ws = torch.rand(e, 2 * up if swiglu else -(-n // 128), k // 128, device=DEV) * 0.1
    q, s = ops.quant_fp8_1x128(torch.randn(rows + 3, k, device=DEV, dtype=torch.bfloat16))
    got = ops.grouped_gemm_fp8_block(q, s, w, ws, offs, swiglu, up)[:rows]
    monkeypatch.setattr(ops, "FP8_STREAM_GROUP_ROWS", 0)
    want = ops.grouped_gemm_fp8_block(q, s, w, ws, offs, swiglu, up)[:rows]
    _close(got, want, 1e-3, 2 ** -7)       # the same sums, rounded once
    ops.check_status()


@pytest.mark.parametrize("used", [3, 200])
def test_grouped_products_chosen_by_the_rows_in_use(used):
    """Any estimate of the rows gives the same result."""
    torch.manual_seed(used)
    e, n, k, cap = 4, 512, 256, 3000
    offs = (torch.arange(e + 1, device=DEV) * used // e).int()
    a, w = torch.randn(cap, k, device=DEV).bfloat16(), (torch.randn(e, n, k, device=DEV) * k ** -0.5).bfloat16()
    want = torch.cat([a[offs[i]: offs[i + 1]].double() @ w[i].double().T for i in range(e)]).float()
    q, s = ops.quant_fp8_1x128(a)
    w8, ws = torch.randn(e, n, k, device=DEV).to(torch.float8_e4m3fn), torch.rand(e, n // 128, k // 128, device=DEV)
    want8 = ops.grouped_gemm_fp8_block(q[:used], s[:used], w8, ws, offs)
    for rows in (None, used, 1, 10 * cap):
        got = ops.grouped_gemm(a, w, offs, rows=rows)
        assert got.shape == (cap, n)
        _close(got[:used], want, 1e-3, 2 ** -8)      # one rounding to bf16
        _close(ops.grouped_gemm_fp8_block(q, s, w8, ws, offs, rows=rows)[:used], want8, 1e-3, 2 ** -7)


@pytest.mark.parametrize("m,n,k", [(1, 130, 128), (33, 1000, 640), (64, 4096, 1024), (65, 260, 384)])
def test_gemm_fp8_block_against_64_bits(m, n, k):
    """Scale rows of a ragged N, K splits, epilogues, on either side of the 64 rows of the weight-streaming kernel."""
    torch.manual_seed(m + n + k)
    q, s = ops.quant_fp8_1x128(torch.randn(m, k, device=DEV, dtype=torch.bfloat16))
    w, ws = torch.randn(n, k, device=DEV).to(torch.float8_e4m3fn), torch.rand(-(-n // 128), k // 128, device=DEV) + 0.5
    full = w.double() * ws.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)
    exact = (q.double() * s.double().repeat_interleave(128, 1)) @ full.T
    bias, res = torch.randn(n, device=DEV).bfloat16(), torch.randn(m, n, device=DEV).bfloat16()
    # fp32 sums of k products of size 1
    _close(ops.gemm_fp8_block(q, s, w, ws, out_dtype=torch.float32), exact.float(), k ** 0.5 * 2 ** -16, 2 ** -16)
    # one rounding to bf16
    _close(ops.gemm_fp8_block(q, s, w, ws, bias, res), (exact + bias.double() + res.double()).float(), 1e-2, 2 ** -8)


@pytest.mark.parametrize("counts,n,k,swiglu", [([0, 5, 64, 65, 0, 16], 512, 256, True), ([3, 40], 130, 128, False),
                                               ([70, 1], 768, 384, True), ([200, 180], 512, 256, True)])
def test_grouped_gemm_fp8_block_against_64_bits(counts, n, k, swiglu):
    """Scale rows of alternating gate and up rows, groups of any size, few rows per group and many."""
    torch.manual_seed(n + k)
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32)
    rows, e = int(offs[-1]), len(counts)
    w = torch.randn(e, n, k, device=DEV).to(torch.float8_e4m3fn)
    r = torch.arange(n)
    up = n // 256 if swiglu else 0
    block = torch.where((r & 8) != 0, up, 0) + (r // 16 * 8 + r % 8) // 128 if swiglu else r // 128
    ws = torch.rand(e, 2 * up if swiglu else -(-n // 128), k // 128, device=DEV) * 0.2 + 0.05
    q, s = ops.quant_fp8_1x128(torch.randn(rows, k, device=DEV, dtype=torch.bfloat16))
    x = q.double() * s.double().repeat_interleave(128, 1)
    full = w.double() * ws.double()[:, block.to(DEV)].repeat_interleave(128, 2)
    exact = torch.cat([x[offs[i]: offs[i + 1]] @ full[i].T for i in range(e)])
    if swiglu:
        gate, upper = exact.view(rows, -1, 2, 8).unbind(2)
        exact = (torch.nn.functional.silu(gate) * upper).reshape(rows, -1)
    # one rounding to bf16, of fp32 sums
    _close(ops.grouped_gemm_fp8_block(q, s, w, ws, offs.to(DEV), swiglu, up), exact.float(), 1e-2, 2 ** -7)


@pytest.mark.parametrize("limit", [1, 7, 40, 300])
def test_few_rows_within_a_limit_of_ctas(limit):
    torch.manual_seed(limit)
    m, n, k = 20, 1000, 2048
    a = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = (torch.randn(n, k, device=DEV) * k ** -0.5).bfloat16()
    # fp32 sums of k products of size k ** -0.5
    _close(ops.gemm(a, w, out_dtype=torch.float32, max_ctas=limit), (a.double() @ w.double().T).float(), k ** 0.5 * 2 ** -22, 0)
    q, s = ops.quant_fp8_1x128(a)
    w8, ws = torch.randn(n, k, device=DEV).to(torch.float8_e4m3fn), torch.rand(8, k // 128, device=DEV) + 0.5
    full = w8.double() * ws.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)
    want = (q.double() * s.double().repeat_interleave(128, 1)) @ full.T
    # fp32 sums of products of size 1: k ** 0.5 of them in size, each off by some 2 ** -24 of the largest part
    _close(ops.gemm_fp8_block(q, s, w8, ws, out_dtype=torch.float32, max_ctas=limit), want.float(), k ** 0.5 * 2 ** -16, 2 ** -16)


@pytest.mark.parametrize("t,h,lat,rope,nope", [(1, 16, 512, 64, 128), (40, 3, 512, 64, 128), (7, 1, 8, 8, 16), (5, 2, 4096, 32, 64),
                                               (9, 2, 260, 64, 128), (6, 2, 512, 64, 100)])
def test_mla_norm_rope_cache(t, h, lat, rope, nope):
    """Latent rows into the cache and the queries' rotated part in place (and shapes for which they are separate kernels)."""
    torch.manual_seed(t)
    q = torch.randn(t, h, nope + rope, device=DEV, dtype=torch.bfloat16)
    kv = torch.randn(t, lat + rope, device=DEV, dtype=torch.bfloat16)
    w = (torch.rand(lat, device=DEV) + 0.5).bfloat16()
    pos = torch.randint(0, 500, (t,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(64)[:t].int()
    if t > 2:
        slots[2] = -1
    cs = ref.build_cos_sin_cache(rope, 512, 10000.0).to(DEV)
    cache = torch.zeros(4, 16, lat + rope, device=DEV, dtype=torch.bfloat16)
    c, s = cs.double()[pos.long()].chunk(2, -1)

    def turned(x):
        x = x.double()
        cc, ss = (c, s) if x.dim() == 2 else (c[:, None], s[:, None])
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * cc - b * ss, b * cc + a * ss], -1).flatten(-2)

    want_q, head = turned(q[..., nope:]), q[..., :nope].clone()
    row = kv[:, :lat].double()
    row = torch.cat([row * torch.rsqrt(row.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double(), turned(kv[:, lat:])], -1)
    got = ops.mla_norm_rope_cache_(q, nope, kv, w, cache, pos, slots.to(DEV), cs, 1e-6)
    # one rounding to bf16
    _close(got, want_q.float(), 1e-3, 2 ** -8)
    assert torch.equal(q[..., :nope], head)
    flat, used = cache.view(64, -1), [i for i in range(t) if slots[i] >= 0]
    _close(flat[slots[used].long()], row[used].float(), 1e-3, 2 ** -8)
    assert int((flat != 0).any(-1).sum()) == len(used)


@pytest.mark.parametrize("t,g,n,k", [(1, 16, 512, 128), (33, 16, 128, 512), (130, 3, 200, 72), (300, 16, 512, 128), (5, 1, 24, 8),
                                     (65, 128, 512, 64)])
@pytest.mark.parametrize("at", [16, 4])
def test_batched_gemm(t, g, n, k, at):
    """Groups read and written where they lie among wider rows (from the fourth element on: an address that the copies do
    not take)."""
    torch.manual_seed(t + n)
    a = torch.randn(t, g, k + 24, device=DEV, dtype=torch.bfloat16)[..., at: at + k]
    w = (torch.randn(g, n, k, device=DEV) * k ** -0.5).bfloat16()
    rows = torch.zeros(t, g, n + 64, device=DEV, dtype=torch.bfloat16)
    out = ops.batched_gemm(a, w, rows[..., :n])
    # one rounding to bf16
    _close(out, torch.einsum("tgk,gnk->tgn", a.double(), w.double()).float(), 1e-3, 2 ** -8)
    assert int(rows[..., n:].abs().max()) == 0


@pytest.mark.parametrize("new,cached", [([1], [0]), ([300, 1, 128, 17], [0, 700, 3, 129]), ([257, 5], [0, 0])])
def test_mla_prefill(new, cached):
    """Latent attention over up-projected rows where they lie, sequences at starts of their own."""
    torch.manual_seed(len(new))
    h, lens = 3, [a + b for a, b in zip(new, cached)]
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + -(-n // 16) * 16)
    kv = torch.randn(starts[-1], h, 256, device=DEV, dtype=torch.bfloat16)
    lat = torch.randn(starts[-1], 576, device=DEV, dtype=torch.bfloat16)
    q = torch.randn(sum(new), h, 192, device=DEV, dtype=torch.bfloat16)
    cu = torch.tensor([0] + new).cumsum(0)
    i32 = dict(dtype=torch.int32, device=DEV)
    out = ops.mla_prefill(q, kv, lat[:, 512:], torch.tensor(starts[:-1], **i32), cu.to(**i32), torch.tensor(lens, **i32), len(new),
                          max(new), 192 ** -0.5)
    for i, n in enumerate(lens):
        rows = slice(starts[i], starts[i] + n)
        k = torch.cat([kv[rows, :, :128], lat[rows, None, 512:].expand(-1, h, -1)], -1).double()
        s = torch.einsum("qhd,khd->hqk", q[cu[i]: cu[i + 1]].double(), k) * 192 ** -0.5
        hidden = torch.arange(n, device=DEV)[None] > cached[i] + torch.arange(new[i], device=DEV)[:, None]
        want = torch.einsum("hqk,khd->qhd", s.masked_fill(hidden, -math.inf).softmax(-1), kv[rows, :, 128:].double())
        # P is rounded to bf16 (2 ** -9 of values up to 4 or so), and so is the result
        _close(out[cu[i]: cu[i + 1]], want.flatten(1).float(), 2e-2, 2 ** -7)


@pytest.mark.parametrize("bs", [8, 16, 64])
@pytest.mark.parametrize("dqk", [128, 192])
def test_prefill_keeps_other_sequences_nans_out(bs, dqk):
    """Rows of a key tile past the end of a sequence take no part, whatever other sequences left in shared memory."""
    torch.manual_seed(bs)
    hq = hk = 8
    lens = [700] * 20 + [3, 17, 133, 250, 129, 8]            # more items than SMs: later ones follow the first
    bad = 20                                                 # sequences whose values are NaN and infinite
    nb = [-(-n // bs) for n in lens]
    kc = torch.randn(sum(nb), hk, bs, dqk, device=DEV, dtype=torch.bfloat16)
    vc = torch.randn(sum(nb), hk, bs, 128, device=DEV, dtype=torch.bfloat16)
    vc[: sum(nb[:bad])] = float("nan")
    vc[: nb[0]] = float("inf")
    bt = torch.zeros(len(lens), max(nb), dtype=torch.int32)
    at = 0
    for i, n in enumerate(nb):
        bt[i, :n] = torch.arange(at, at + n)
        at += n
    cu = torch.tensor([0] + lens).cumsum(0).int()
    q = torch.randn(sum(lens), hq * dqk, device=DEV, dtype=torch.bfloat16)
    out = ops.gqa_prefill(q, kc, vc, bt.to(DEV), cu.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), len(lens),
                          max(lens), hq, dqk ** -0.5)
    assert not torch.isfinite(out[: cu[bad]].float()).any()
    tail = slice(int(cu[bad]), None)
    want = ref.paged_attention(q[tail].cpu(), kc.cpu(), vc.cpu(), bt[bad:], cu[bad:] - cu[bad],
                               torch.tensor(lens[bad:], dtype=torch.int32), hq, dqk ** -0.5, True, 0, False, 0)
    _close(out[tail], want, 2e-2, 2e-2)


@pytest.mark.parametrize("bs", [8, 16, 64, 128])
@pytest.mark.parametrize("dqk,hq,hk", [(128, 8, 2), (128, 3, 1), (192, 4, 4)])
@pytest.mark.parametrize("causal", [True, False])
def test_prefill_keeps_the_rest_of_the_last_page_out(bs, dqk, hq, hk, causal):
    """What an earlier owner left behind a sequence's last key takes no part, be it infinite or NaN."""
    lens, new = [3, 17, 133, 250, 129, 8, 260, 120], [3, 16, 133, 1, 129, 8, 200, 2]
    q, kc, vc, bt, cu, sl = _paged_setup(lens, new, hq, hk, dqk, bs, dv=128, seed=bs)
    want = ref.paged_attention(q, kc, vc, bt, cu, sl, hq, dqk ** -0.5, causal, 0)
    for i, n in enumerate(lens):
        if n % bs:
            last = int(bt[i, n // bs])
            kc[last, :, n % bs:], vc[last, :, n % bs:] = float("nan"), float("nan") if i % 2 else float("-inf")
    got = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV), len(lens), max(new), hq,
                          dqk ** -0.5, causal)
    # P and the result are rounded to bf16 (2 ** -9 each) of values up to about 4
    _close(got, want, 2e-2, 2e-2)


@pytest.mark.parametrize("shift,scale", [(0, 192 ** -0.5), (4, 192 ** -0.5), (0, -0.07)])
def test_mla_prefill_refuses_what_its_copies_do_not_take(shift, scale):
    """Rotated parts off a 16-byte boundary and negative scales are the caller's to repack."""
    q, kv = (torch.randn(8, 2, n, device=DEV, dtype=torch.bfloat16) for n in (192, 256))
    pe = torch.randn(8, 64 + 8, device=DEV, dtype=torch.bfloat16)[:, shift: shift + 64]
    i32 = dict(dtype=torch.int32, device=DEV)
    out = ops.mla_prefill(q, kv, pe, torch.zeros(1, **i32), torch.tensor([0, 8], **i32), torch.tensor([8], **i32), 1, 8, scale)
    assert (out is None) == (shift != 0 or scale < 0)


@pytest.mark.parametrize("hq,hk", [(8, 2), (3, 1)])
@pytest.mark.parametrize("causal", [True, False])
def test_prefill_rows_without_keys_are_zero(hq, hk, causal):
    """Sequences without keys (another rank's, or a padded one), and rows that lie ahead of the first key."""
    lens, new = [0, 40, 0, 3, 0, 150], [5, 40, 200, 300, 1, 260]
    q, kc, vc, bt, cu, sl = _paged_setup(lens, new, hq, hk, 128, 16, seed=hq)
    junk = [torch.full((sum(new), hq * 128), 7.0, device=DEV, dtype=torch.bfloat16) for _ in range(4)]
    del junk                                   # what the result's memory holds before
    got, lse = ops.gqa_prefill(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cu.to(DEV), sl.to(DEV), len(lens), max(new), hq,
                               128 ** -0.5, causal, 0, True)
    got, lse = got.cpu().view(-1, hq, 128), lse.cpu()
    for i, n in enumerate(lens):
        for r in range(new[i]):
            row, seen = int(cu[i]) + r, max(0, n - new[i] + r + 1) if causal else n
            if seen == 0:
                assert not got[row].any() and (lse[row] == -math.inf).all()
            elif r % 37 == 0 or r == new[i] - 1:
                k, v = (c[bt[i].long()].transpose(1, 2).flatten(0, 1)[:seen].double() for c in (kc, vc))
                k, v = (x.repeat_interleave(hq // hk, 1) for x in (k, v))
                s = torch.einsum("hd,khd->hk", q[row].view(hq, 128).double(), k) * 128 ** -0.5
                _close(got[row], torch.einsum("hk,khd->hd", s.softmax(-1), v), 2e-2, 2e-2)
                _close(lse[row], s.logsumexp(-1), 2e-2, 1e-2)


@pytest.mark.parametrize("page", [8, 24])
def test_mla_prefill_keeps_other_sequences_out(page):
    """Sequences that start at any page, each followed by one with NaN and infinite values."""
    torch.manual_seed(page)
    h, lens, new = 2, [8, 3, 133, 40, 250, 5, 129], [8, 3, 133, 40, 20, 5, 129]
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + -(-n // page) * page)
    i32 = dict(dtype=torch.int32, device=DEV)
    kv = torch.randn(starts[-1], h, 256, device=DEV, dtype=torch.bfloat16)
    lat = torch.randn(starts[-1], 576, device=DEV, dtype=torch.bfloat16)
    q = torch.randn(sum(new), h, 192, device=DEV, dtype=torch.bfloat16)
    cu = torch.tensor([0] + new).cumsum(0)
    args = (cu.to(**i32), torch.tensor(lens, **i32), len(new), max(new), 192 ** -0.5)
    for sound in range(2):                       # of every two neighbours one is sound
        bad = kv.clone()
        for i, n in enumerate(lens):
            bad[starts[i] + n: starts[i + 1]] = float("nan")
            if i % 2 != sound:
                bad[starts[i]: starts[i + 1]] = float("nan") if i % 4 < 2 else float("inf")
        out = ops.mla_prefill(q, bad, lat[:, 512:], torch.tensor(starts[:-1], **i32), *args)
        for i, n in enumerate(lens):
            if i % 2 != sound:
                continue
            rows = slice(starts[i], starts[i] + n)
            k = torch.cat([kv[rows, :, :128], lat[rows, None, 512:].expand(-1, h, -1)], -1).double()
            s = torch.einsum("qhd,khd->hqk", q[cu[i]: cu[i + 1]].double(), k) * 192 ** -0.5
            hidden = torch.arange(n, device=DEV)[None] > n - new[i] + torch.arange(new[i], device=DEV)[:, None]
            want = torch.einsum("hqk,khd->qhd", s.masked_fill(hidden, -math.inf).softmax(-1), kv[rows, :, 128:].double())
            _close(out[cu[i]: cu[i + 1]], want.flatten(1).float(), 2e-2, 2 ** -7)


@pytest.mark.parametrize("t,hq,hk,d,rot,neox", [(1, 32, 4, 128, 128, True), (37, 3, 1, 16, 16, True), (300, 5, 2, 64, 64, True),
                                                (9, 2, 2, 256, 256, True), (3, 1, 1, 512, 512, True),
                                                (17, 4, 2, 128, 64, True), (5, 4, 2, 96, 96, True), (6, 4, 2, 128, 128, False)])
@pytest.mark.parametrize("normed", [True, False])
def test_rope_cache_gqa_norm(t, hq, hk, d, rot, neox, normed):
    """Norm per head, rotation and cache rows in one pass (and heads for which they are separate kernels)."""
    torch.manual_seed(t + d)
    bs = 16
    qkv = torch.randn(t, (hq + 2 * hk) * d, device=DEV, dtype=torch.bfloat16) * 3
    q, k, v = qkv.split([hq * d, hk * d, hk * d], 1)
    w = [(torch.rand(d, device=DEV) + 0.5).bfloat16() for _ in range(2)]
    eps = 1e-3
    pos = torch.randint(0, 1000, (t,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(20 * bs)[:t].to(torch.int32)
    if t > 3:
        slots[3] = -1
    cs = ref.build_cos_sin_cache(rot, 1024, 10000.0).to(DEV)

    def exact(x, g):
        x = x.double().view(t, -1, d)
        if normed:
            x = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * g.double()
        c, s = cs.double()[pos.long()][:, None].chunk(2, -1)
        r = x[..., :rot]
        a, b = r.chunk(2, -1) if neox else (r[..., 0::2], r[..., 1::2])
        u, y = a * c - b * s, b * c + a * s
        r = torch.cat([u, y], -1) if neox else torch.stack([u, y], -1).flatten(-2)
        return torch.cat([r, x[..., rot:]], -1)

    want_q, want_k, want_v = exact(q, w[0]), exact(k, w[1]), v.reshape(t, hk, d).clone()
    kc = torch.zeros(20, hk, bs, d, device=DEV, dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    got = ops.rope_cache_gqa_(q, k, v, kc, vc, pos, slots.to(DEV), cs, d, rot, neox, (*w, eps) if normed else None)
    # one rounding to bf16, of values up to some 12 times the weight; a second one where the norm is a kernel of its own
    _close(got.view(t, hq, d), want_q.float(), 2e-2, 2 ** -8)
    for i, s in enumerate(slots.tolist()):
        if s >= 0:
            _close(kc[s // bs, :, s % bs], want_k[i].float(), 2e-2, 2 ** -8)
            assert torch.equal(vc[s // bs, :, s % bs], want_v[i])
    written = (slots >= 0).sum().item()
    assert int((vc != 0).any(-1).any(1).sum()) == written


@pytest.mark.parametrize("t,hq,hk,d", [(5, 64, 8, 128), (3, 65, 1, 128), (2, 130, 2, 64), (1, 40, 30, 256)])
@pytest.mark.parametrize("normed", [True, False])
def test_rope_cache_gqa_many_heads(t, hq, hk, d, normed):
    """More heads than a CTA takes at once."""
    test_rope_cache_gqa_norm(t, hq, hk, d, d, True, normed)


def test_rope_cache_gqa_and_cache_write():
    t, hq, hk, d, bs = 29, 8, 2, 128, 16
    qkv = torch.randn(t, (hq + 2 * hk) * d, device=DEV, dtype=torch.bfloat16)
    q, k, v = qkv[:, : hq * d], qkv[:, hq * d: (hq + hk) * d], qkv[:, (hq + hk) * d:]
    pos = torch.randint(0, 1000, (t,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(10 * bs)[:t].to(torch.int32)
    slots[3] = -1
    cs = ref.build_cos_sin_cache(d, 1024, 500000.0).to(DEV)
    kc = torch.zeros(10, hk, bs, d, device=DEV, dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    kc_ref, vc_ref = kc.cpu().clone(), vc.cpu().clone()
    qr, kr = ref.rope_qk(q.cpu(), k.cpu(), pos.cpu(), cs.cpu(), d, d, True)
    ref.gqa_cache_write(kr, v.cpu(), kc_ref, vc_ref, slots)
    ops.rope_cache_gqa_(q, k, v, kc, vc, pos, slots.to(DEV), cs, d, d, True)
    _close(q, qr, 2e-2, 2e-2)
    _close(kc, kc_ref, 2e-2, 2e-2)
    _close(vc, vc_ref, 0, 0)
    kc2, vc2 = torch.zeros_like(kc), torch.zeros_like(vc)
    ops.gqa_cache_write(k, v, kc2, vc2, slots.to(DEV))
    kc3, vc3 = torch.zeros_like(kc_ref), torch.zeros_like(vc_ref)
    ref.gqa_cache_write(k.cpu(), v.cpu(), kc3, vc3, slots)
    _close(kc2, kc3, 0, 0)
    _close(vc2, vc3, 0, 0)


def test_mla_kv_rmsnorm_rope_cache():
    t, l, r, bs = 21, 512, 64, 16
    kv = torch.randn(t, l + r, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(l, device=DEV, dtype=torch.bfloat16)
    pos = torch.randint(0, 900, (t,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(4 * bs)[:t].to(torch.int32)
    cs = ref.build_cos_sin_cache(r, 1024, 10000.0).to(DEV)
    cache = torch.zeros(4, bs, l + r, device=DEV, dtype=torch.bfloat16)
    cache_ref = cache.cpu().clone()
    a = ops.mla_kv_rmsnorm_rope_cache(kv[:, :l], kv[:, l:], w, cache, pos, slots.to(DEV), cs, 1e-6, False, True)
    b = ops.mla_kv_rmsnorm_rope_cache(kv[:, :l].cpu(), kv[:, l:].cpu(), w.cpu(), cache_ref, pos.cpu(), slots,
                                      cs.cpu(), 1e-6, False, True)
    _close(cache, cache_ref, 3e-2, 2e-2)
    _close(a[0], b[0], 3e-2, 2e-2)
    _close(a[1], b[1], 3e-2, 2e-2)


# ------------------------------------------------------------------ sampling
def test_argmax_and_greedy_sample():
    torch.manual_seed(0)
    logits = torch.randn(33, 128256, device=DEV, dtype=torch.float32)
    want = logits.argmax(-1).to(torch.int32)
    assert torch.equal(ops.argmax(logits), want)
    assert torch.equal(ops.argmax(logits.bfloat16()), logits.bfloat16().float().argmax(-1).to(torch.int32))
    t = torch.zeros(33, device=DEV)
    got = ops.sample(logits, t, torch.zeros(33, dtype=torch.int32, device=DEV), torch.ones(33, device=DEV),
                     torch.arange(33, device=DEV), torch.zeros(1, dtype=torch.int64, device=DEV))
    assert torch.equal(got, want)


def test_sample_respects_top_k_top_p_and_distribution():
    torch.manual_seed(1)
    v, n = 1000, 4096
    base = torch.randn(v, device=DEV) * 2
    logits = base.unsqueeze(0).repeat(n, 1).contiguous()
    temp = torch.full((n,), 0.8, device=DEV)
    topk = torch.full((n,), 20, dtype=torch.int32, device=DEV)
    topp = torch.full((n,), 0.9, device=DEV)
    seeds = torch.arange(n, device=DEV, dtype=torch.int64) * 7919 + 13
    step = torch.zeros(1, dtype=torch.int64, device=DEV)
    got = ops.sample(logits, temp, topk, topp, seeds, step).long().cpu()
    masked = ref.apply_top_k_top_p((base / 0.8).unsqueeze(0).cpu(), torch.tensor([20]), torch.tensor([0.9]))[0]
    allowed = torch.isfinite(masked)
    assert allowed[got].all(), "sampled a token outside the top-k/top-p set"
    probs = masked.softmax(-1)
    freq = torch.bincount(got, minlength=v).float() / n
    assert (freq - probs).abs().max() < 0.04
    # a different step offset gives different draws; the same offset repeats them
    again = ops.sample(logits, temp, topk, topp, seeds, step).long().cpu()
    assert torch.equal(again, got)
    other = ops.sample(logits, temp, topk, topp, seeds, step + 1).long().cpu()
    assert (other != got).float().mean() > 0.3


def _philox_u(seed, row, groups):
    """Uniform numbers (0, 1] of the sampling kernel's draw: Philox4x32-10, a counter per four logits."""
    import numpy as np
    c = [np.arange(groups, dtype=np.uint64), np.zeros(groups, np.uint64), np.zeros(groups, np.uint64),
         np.full(groups, row, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        lo, hi = np.uint64(0xFFFFFFFF), np.uint64(32)
        c = [(b >> hi) ^ c[1] ^ np.uint64(k0), b & lo, (a >> hi) ^ c[3] ^ np.uint64(k1), a & lo]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return (torch.from_numpy((np.stack(c, 1).reshape(-1) >> np.uint64(8)).astype(np.float64)) + 1) / 2 ** 24


@pytest.mark.parametrize("v,dtype,pad", [(1, torch.float32, 0), (7, torch.float32, 1), (1000, torch.bfloat16, 0),
                                         (4097, torch.float32, 3), (128256, torch.float32, 0),
                                         (151936, torch.bfloat16, 8), (410001, torch.float32, 3)])
def test_sample_draws_the_best_race_among_the_kept_logits(v, dtype, pad):
    """Slices with remainders, rows off 16-byte boundaries, a row too long for shared memory, equal logits; rows take
    turns in top-k, top-p, both, neither."""
    torch.manual_seed(v)
    n = 10
    logits = (torch.randn(n, v + pad, device=DEV) * 2).to(dtype)[:, :v]
    logits[8:] = 1.5                                            # all equal: the chosen bin holds the whole row
    row = torch.arange(n, device=DEV)
    temp = 0.3 + 0.15 * row
    top_k = torch.where(row % 4 == 1, 50, torch.where(row % 4 == 3, 1, 0)).int()
    top_p = torch.where(row % 4 >= 2, 0.9, 1.0).float()
    top_p[9], top_k[5], top_p[6] = 0.5, v, 0.0
    seeds = torch.arange(n, device=DEV) * 0x123456789 + 5
    got = ops.sample(logits, temp, top_k, top_p, seeds, None).tolist()
    for i in range(n):
        x = logits[i].double().cpu()
        k, p, t = int(top_k[i]), float(top_p[i]), float(temp[i])
        if p == 0.0:
            assert got[i] == int(x.argmax())
            continue
        order = x.sort(descending=True).values
        floor = order[k - 1] if 0 < k < v else order[-1]
        if p < 1:
            w = torch.where(order >= floor, ((order - order[0]) / t).exp(), 0.0).cumsum(0)
            # 1e-5: fp32 sums of positive numbers and the 2^-22 of exp2
            lowest = order[min(v - 1, int((w < p * w[-1] * (1 + 1e-5)).sum()))]
            surest = order[int((w < p * w[-1] * (1 - 1e-5)).sum())]
        else:
            lowest = surest = floor
        u = _philox_u(int(seeds[i]), i, -(-v // 4))[:v]
        score = x / t - (-u.log()).clamp_min(1e-30).log()
        assert x[got[i]] >= max(lowest, floor)
        # fp32: x / t within 2^-22 of it, a logarithm within 2^-20 (u near 1 keeps 24 bits of it)
        best = float(score[x >= max(surest, floor)].max())
        e = float(-u[got[i]].log())
        assert float(score[got[i]]) >= best - 1e-4 - 2e-6 / max(e, 1e-7)


@pytest.mark.parametrize("v,dtype,pad", [(8192, torch.float32, 0), (8193, torch.float32, 3), (8190, torch.bfloat16, 2),
                                         (49152, torch.float32, 0), (49154, torch.float32, 2), (32000, torch.bfloat16, 0)])
def test_sample_on_one_four_and_eight_ctas(v, dtype, pad):
    """The same draw on either side of the lengths at which a row takes more CTAs."""
    test_sample_draws_the_best_race_among_the_kept_logits(v, dtype, pad)


@pytest.mark.parametrize("v", [5, 1000, 20000, 128256])
def test_sample_rows_without_numbers(v):
    """NaN and infinite logits give a token of the vocabulary, with and without thresholds."""
    rows = [float("nan"), float("-inf"), float("inf")]
    logits = torch.tensor(rows, device=DEV).repeat_interleave(4).view(-1, 1).repeat(1, v)
    logits = torch.cat([logits, torch.full((4, v), float("-inf"), device=DEV)])
    logits[12:, v // 2] = 0.0                                   # one token possible
    n = logits.shape[0]
    top_k = torch.tensor([0, 3, 0, 3] * (n // 4), dtype=torch.int32, device=DEV)
    top_p = torch.tensor([1.0, 1.0, 0.9, 0.9] * (n // 4), device=DEV)
    got = ops.sample(logits, torch.full((n,), 0.7, device=DEV), top_k, top_p, torch.arange(n, device=DEV), None)
    assert got.min() >= 0 and got.max() < v
    assert (got[:4] == 0).all() and (got[12:] == v // 2).all()


# --------------------------------------------------------------------- MoE
@pytest.mark.parametrize("e,k,sigmoid,groups,bias", [(64, 6, False, (1, 1), False), (128, 8, False, (1, 1), False),
                                                      (256, 8, True, (8, 4), True), (8, 2, True, (4, 2), False)])
def test_moe_topk(e, k, sigmoid, groups, bias):
    torch.manual_seed(0)
    t = 77
    logits = torch.randn(t, e, device=DEV)
    b = (torch.randn(e, device=DEV) * 0.1) if bias else None
    ids, w = ops.moe_topk(logits, b, k, sigmoid, groups[0], groups[1], True, 2.5)
    ids_r, w_r = ref.moe_topk(logits.cpu(), b.cpu() if bias else None, k, sigmoid, groups[0], groups[1], True, 2.5)
    # same selected set (order of equal scores may differ) and same weights per expert
    assert torch.equal(ids.cpu().sort(-1).values, ids_r.sort(-1).values)
    got = torch.zeros(t, e).scatter_(1, ids.cpu().long(), w.cpu())
    want = torch.zeros(t, e).scatter_(1, ids_r.long(), w_r)
    torch.testing.assert_close(got, want, atol=1e-5, rtol=1e-4)


def test_fused_moe_layer_single_gpu_matches_cpu_reference():
    from omni_npu_b200.layers.moe import FusedMoE
    torch.manual_seed(1)
    kw = dict(num_experts=16, top_k=4, hidden_size=256, intermediate_size=128, num_shared_experts=1,
              renormalize=True, max_tokens=512)
    gpu = FusedMoE(dtype=torch.bfloat16, device=DEV, **kw)
    for p in gpu.parameters():
        p.data.normal_(0, 0.05)
    cpu = FusedMoE(dtype=torch.bfloat16, **kw)
    cpu.load_state_dict({k_: v.cpu() for k_, v in gpu.state_dict().items()})
    for t in (1, 37, 300):
        x = torch.randn(t, 256, device=DEV, dtype=torch.bfloat16)
        _close(gpu(x), cpu(x.cpu()), 3e-2, 3e-2)
    # inactive (padded) rows: ids of -1 must contribute nothing and must not fault
    x = torch.randn(8, 256, device=DEV, dtype=torch.bfloat16)
    w = torch.full((8, 4), 0.25, device=DEV)
    ids = torch.randint(0, 16, (8, 4), device=DEV, dtype=torch.int32)
    ids[5:] = -1
    out = gpu._routed(x, w, ids)
    sh = gpu.shared_experts(x)
    _close(out[5:], sh[5:], 2e-2, 2e-2)


# --------------------------------------------------------------------- MLA
@pytest.mark.parametrize("n_heads,splits,q_len", [(16, 1, 1), (16, 3, 1), (128, 2, 1), (8, 2, 2)])
def test_mla_decode(n_heads, splits, q_len):
    torch.manual_seed(3)
    bs, seq_lens = 16, [5, 64, 200, 1031]
    b = len(seq_lens)
    max_blocks = max((s + bs - 1) // bs for s in seq_lens) + 1
    nblocks = b * max_blocks + 2
    bt = torch.randperm(nblocks)[: b * max_blocks].view(b, max_blocks).to(torch.int32)
    cache = torch.randn(nblocks, bs, 576).bfloat16()
    q = (torch.randn(b * q_len, n_heads * 576) * 0.3).bfloat16()
    sl = torch.tensor(seq_lens, dtype=torch.int32)
    want, want_lse = ref.mla_decode(q, cache, bt, sl, b, q_len, n_heads, 0.07, None, True)
    got, lse = ops.mla_decode(q.to(DEV), cache.to(DEV), bt.to(DEV), sl.to(DEV), b, n_heads, 0.07, q_len,
                              splits=splits, return_lse=True)
    _close(got, want, 2e-2, 2e-2)
    _close(lse, want_lse, 2e-2, 2e-2)


def test_mla_decode_sparse_selection():
    torch.manual_seed(4)
    bs, n_heads, topk = 16, 16, 128
    seq_lens = [300, 90]
    b = len(seq_lens)
    max_blocks = 20
    bt = torch.randperm(b * max_blocks)[: b * max_blocks].view(b, max_blocks).to(torch.int32)
    cache = torch.randn(b * max_blocks, bs, 576).bfloat16()
    q = (torch.randn(b, n_heads * 576) * 0.3).bfloat16()
    sl = torch.tensor(seq_lens, dtype=torch.int32)
    sel = torch.full((b, topk), -1, dtype=torch.int32)
    sel[0] = torch.randperm(300)[:topk].to(torch.int32)
    sel[1, :90] = torch.randperm(90).to(torch.int32)
    sel[1, 7] = -1
    want = ref.mla_decode(q, cache, bt, sl, b, 1, n_heads, 0.07, sel)
    got = ops.mla_decode(q.to(DEV), cache.to(DEV), bt.to(DEV), sl.to(DEV), b, n_heads, 0.07, 1, sel.to(DEV), splits=2)
    _close(got, want, 2e-2, 2e-2)


@pytest.mark.parametrize("bs", [8, 16, 32, 64, 128])
@pytest.mark.parametrize("seq_lens,n_heads,q_len", [([1, 31, 32, 33, 7], 16, 1), ([64, 95, 96, 97, 128, 130], 16, 1),
                                                    ([159, 160, 161, 2000, 5], 20, 1), ([2, 40, 162], 16, 2)])
def test_mla_decode_tiles(bs, seq_lens, n_heads, q_len):
    """Pages smaller and larger than a tile of 32 keys, lengths around a tile, a tile per group and a ring, splits by rule;
    what other kernels left in shared memory and in the rest of a page that no copy brings takes no part."""
    torch.manual_seed(bs)
    b = len(seq_lens)
    max_blocks = max(-(-n // bs) for n in seq_lens) + 1
    nblocks = b * max_blocks + 2
    bt = torch.randperm(nblocks)[: b * max_blocks].view(b, max_blocks).to(torch.int32)
    cache = torch.randn(nblocks, bs, 576).bfloat16()
    q = (torch.randn(b * q_len, n_heads * 576) * 0.3).bfloat16()
    sl = torch.tensor(seq_lens, dtype=torch.int32)
    want, want_lse = ref.mla_decode(q, cache, bt, sl, b, q_len, n_heads, 0.07, None, True)
    # NaN in the shared memory of every SM first
    junk = torch.full((100, 16, 576), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops.mla_decode(torch.zeros(300, 16 * 576, device=DEV, dtype=torch.bfloat16), junk,
                   torch.arange(10, device=DEV, dtype=torch.int32).repeat(300, 1),
                   torch.full((300,), 160, device=DEV, dtype=torch.int32), 300, 16, 0.07, splits=1)
    got, lse = ops.mla_decode(q.to(DEV), cache.to(DEV), bt.to(DEV), sl.to(DEV), b, n_heads, 0.07, q_len, return_lse=True)
    _close(got, want, 2e-2, 2e-2)
    _close(lse, want_lse, 2e-2, 2e-2)


@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("add", [False, True])
def test_rms_norm_quant_fused(kind, add):
    torch.manual_seed(11)
    t, h = 37, 4096
    x = torch.randn(t, h, device=DEV, dtype=torch.bfloat16)
    w = (torch.rand(h, device=DEV) + 0.5).bfloat16()
    res = torch.randn(t, h, device=DEV, dtype=torch.bfloat16) if add else None
    res_ref = res.cpu().clone() if add else None
    q, s, y = ops.rms_norm_quant(x, w, 1e-6, res, kind, want_bf16=True)
    q0, s0, y0 = ref.rms_norm_quant(x.cpu(), w.cpu(), 1e-6, res_ref, kind, True)
    if add:
        _close(res, res_ref, 1e-2, 1e-2)
    _close(y, y0, 2e-2, 2e-2)
    _close(s, s0, 1e-6, 2e-2)
    # the quantised row must reproduce the normalised row to within one quantisation step
    deq = q.float().cpu() * s.cpu().unsqueeze(-1)
    step = s.cpu().unsqueeze(-1) * (1.0 if kind == "int8" else 32.0)
    assert ((deq - y.float().cpu()).abs() <= step + 1e-3).all()


@pytest.mark.parametrize("kind", ["int8", "fp8"])
def test_silu_and_mul_quant_fused(kind):
    torch.manual_seed(12)
    t, i = 19, 14336
    x = torch.randn(t, 2 * i, device=DEV, dtype=torch.bfloat16)
    q, s = ops.silu_and_mul_quant(x, kind)
    q0, s0 = ref.silu_and_mul_quant(x.cpu(), kind)
    _close(s, s0, 1e-6, 2e-2)
    y = ops.silu_and_mul(x).float().cpu()
    deq = q.float().cpu() * s.cpu().unsqueeze(-1)
    step = s.cpu().unsqueeze(-1) * (1.0 if kind == "int8" else 32.0)
    assert ((deq - y).abs() <= step + 1e-3).all()


@pytest.mark.parametrize("mode", ["decode", "decode_mtp", "prefill"])
def test_dsa_indexer_scores_and_topk(mode):
    """Indexer on tcgen05 + radix select against the dense fp32 reference: same scores, and the
    selected set is a valid top-k (every selected score >= every unselected one)."""
    torch.manual_seed(21)
    bs, h, topk = 16, 64, 256
    if mode == "prefill":
        ctx, q_lens = [700, 130, 1500], [700, 100, 333]
    elif mode == "decode":
        ctx, q_lens = [5, 257, 900, 2049], [1, 1, 1, 1]
    else:
        ctx, q_lens = [300, 1025, 64], [2, 2, 2]
    b = len(ctx)
    max_blocks = max((c + bs - 1) // bs for c in ctx) + 2
    nblocks = b * max_blocks + 3
    bt = torch.randperm(nblocks)[: b * max_blocks].view(b, max_blocks).to(torch.int32)
    cache = (torch.randn(nblocks, bs, 128) * 0.5).bfloat16()
    t = sum(q_lens)
    q = (torch.randn(t, h, 128) * 0.5).bfloat16()
    w = torch.randn(t, h) * 0.1
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    pos = torch.cat([torch.arange(c - n, c) for c, n in zip(ctx, q_lens)]).to(torch.int32)
    uniform = mode != "prefill"
    want_sel, want_sc = ref.dsa_indexer_topk(q, w, cache, bt, pos, b, topk, None if uniform else cu, q_lens[0], True)
    sel, sc = ops.dsa_indexer_topk(q.to(DEV), w.to(DEV), cache.to(DEV), bt.to(DEV), pos.to(DEV), b, topk,
                                   None if uniform else cu.to(DEV), q_lens[0], max_ctx=max(ctx),
                                   max_q=max(q_lens), return_scores=True)
    sel, sc = sel.cpu(), sc.cpu()
    for i in range(t):
        n = int(pos[i]) + 1
        assert torch.allclose(sc[i, :n], want_sc[i, :n], rtol=2e-2, atol=2e-2), (mode, i)
        got = sel[i][sel[i] >= 0].long()
        assert got.numel() == min(topk, n) and got.unique().numel() == got.numel() and int(got.max()) < n
        if n > topk:
            chosen = torch.zeros(n, dtype=torch.bool)
            chosen[got] = True
            assert sc[i, :n][chosen].min() >= sc[i, :n][~chosen].max()


@pytest.mark.parametrize("m,n,k", [(128, 256, 512), (300, 1000, 1024), (8, 4096, 7168), (2048, 2500, 512)])
def test_gemm_fp8_block_scaled(m, n, k):
    """128 x 128 block-scaled weights, per-token-per-128 activations (DeepSeek-V3 checkpoint format)."""
    from omni_npu_b200.layers.quant_fp8 import fp8_block_gemm, quantize_weight_block
    torch.manual_seed(31)
    x = torch.randn(m, k, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(n, k, device=DEV, dtype=torch.float32) * 0.05
    # per-block magnitudes differ by orders of magnitude, so a missing or misplaced scale shows
    w = w * torch.logspace(-2, 2, (k // 128)).to(DEV).repeat_interleave(128)[None, :]
    wq, ws = quantize_weight_block(w)
    xq, xs = ops.quant_fp8_1x128(x)
    bias = torch.randn(n, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(m, n, device=DEV, dtype=torch.bfloat16)
    want = ref.gemm_fp8_block(xq.cpu(), xs.cpu(), wq.cpu(), ws.cpu(), bias.cpu(), res.cpu(), torch.float32)
    got = ops.gemm_fp8_block(xq, xs, wq, ws, bias, res, torch.float32)
    _close(got, want, 2e-3 * float(want.abs().max()), 2e-3)
    got16 = fp8_block_gemm(x, wq, ws, bias, res)
    assert got16.dtype == torch.bfloat16
    _close(got16, want, 2e-2 * float(want.abs().max()), 2e-2)


@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("swiglu", [False, True])
def test_grouped_gemm_fp8_block_scaled(swiglu, large):
    """Expert GEMM on block-scaled e4m3 weights; with SwiGLU the gate / up rows are interleaved in groups
    of 8 while their scale blocks stay in checkpoint order (gate blocks, then up blocks)."""
    from omni_npu_b200.layers.quant_fp8 import quantize_weight_block
    torch.manual_seed(41)
    e, k, inter = 4, 512, 256
    n = 2 * inter if swiglu else 384
    counts = [130, 0, 7, 300]
    if large:                       # enough 128 x 256 tiles for the two-warp-group variant
        inter = 512
        n = 2 * inter if swiglu else 1000
        counts = [1300, 0, 700, 3000]
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32)
    rows = int(offs[-1])
    x = torch.randn(rows + 50, k, device=DEV, dtype=torch.bfloat16)          # rows past the last expert are unused
    xq, xs = ops.quant_fp8_1x128(x)
    wq = torch.empty(e, n, k, dtype=torch.float8_e4m3fn, device=DEV)
    up0 = (inter + 127) // 128
    ws = torch.empty(e, (2 * up0) if swiglu else (n + 127) // 128, k // 128, device=DEV)
    for i in range(e):
        w = torch.randn(n, k, device=DEV) * 0.05 * torch.logspace(-1, 1, k // 128, device=DEV).repeat_interleave(128)
        if swiglu:
            qg, sg = quantize_weight_block(w[:inter])
            qu, su = quantize_weight_block(w[inter:])
            j = torch.arange(inter, device=DEV)
            wq[i, (j // 8) * 16 + j % 8] = qg
            wq[i, (j // 8) * 16 + 8 + j % 8] = qu
            ws[i, :up0], ws[i, up0:] = sg, su
        else:
            wq[i], ws[i] = quantize_weight_block(w)
    want = ref.grouped_gemm_fp8_block(xq.cpu(), xs.cpu(), wq.cpu(), ws.cpu(), offs, swiglu, up0 if swiglu else 0)
    got = ops.grouped_gemm_fp8_block(xq, xs, wq, ws, offs.to(DEV), swiglu, up0 if swiglu else 0)
    scale = float(want[:rows].float().abs().max())
    _close(got[:rows], want[:rows], 2e-2 * scale, 2e-2)


def test_fused_moe_layer_with_block_scaled_fp8_experts():
    """MoE layer whose experts stay in block-scaled e4m3 on the GPU (grouped block-scaled kernel with the
    SwiGLU epilogue) against the same layer with the weights expanded to fp32 on the CPU."""
    from omni_npu_b200.layers.moe import FusedMoE
    from omni_npu_b200.layers.quant_fp8 import quantize_weight_block
    torch.manual_seed(2)
    e, k, h, inter = 8, 2, 256, 256
    kw = dict(num_experts=e, top_k=k, hidden_size=h, intermediate_size=inter, renormalize=True, max_tokens=512,
              quant="fp8")
    gpu = FusedMoE(dtype=torch.bfloat16, device=DEV, **kw)
    cpu = FusedMoE(dtype=torch.float32, **kw)
    gate_w = torch.randn(e, h) * 0.3
    gpu.gate.weight.data.copy_(gate_w.to(DEV))
    cpu.gate.weight.data.copy_(gate_w)
    for i in range(e):
        for shard, shape, pname, sname in (("gate", (inter, h), "w13", "w13_scale"), ("up", (inter, h), "w13", "w13_scale"),
                                           ("down", (h, inter), "w2", "w2_scale")):
            wq, ws = quantize_weight_block(torch.randn(*shape) * 0.05 * torch.logspace(-0.5, 0.5, shape[0]).unsqueeze(1))
            for layer in (gpu, cpu):
                layer.weight_loader(getattr(layer, pname), wq, i, shard)
                layer.weight_loader(getattr(layer, sname), ws, i, shard)
    gpu.process_weights_after_loading()
    cpu.process_weights_after_loading()
    assert gpu.w13.dtype == torch.float8_e4m3fn and cpu.w13.dtype == torch.float32
    for t in (3, 200):
        x = torch.randn(t, h, device=DEV, dtype=torch.bfloat16)
        want = cpu(x.cpu().float())
        _close(gpu(x), want, 5e-2 * float(want.abs().max()), 5e-2)


def test_bounded_wait_gives_up_and_leaves_the_context_usable():
    """A flag that nothing sets: the wait runs out after its poll limit, the kernel reports status 5
    and returns; the next kernels run normally.  A flag that is already set returns at once."""
    from omni_npu_b200.parallel.symm_mem import wait_probe
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    polls = wait_probe(flag, want=1, max_polls=20000)
    assert polls == 20001
    with pytest.raises(RuntimeError, match="status 5"):
        ops.check_status()
    ops.check_status()                                   # the status word was cleared by the report
    flag.fill_(3)
    assert wait_probe(flag, want=2, max_polls=20000) == 0
    ops.check_status()
    a = torch.randn(64, 128, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(32, 128, device=DEV, dtype=torch.bfloat16)
    _close(ops.gemm(a, w), a.float().cpu() @ w.float().cpu().t(), 2e-1, 2e-2)


def test_ep_dispatch_quantising_scatter_matches_quantise_after_arrival():
    """Expert-parallel dispatch that quantises the rows to e4m3 (one scale per 128 columns) inside the
    scatter kernel: bit-identical to scattering bf16 rows and quantising them afterwards."""
    from omni_npu_b200.layers.moe import _solo_group
    from omni_npu_b200.layers.moe_dispatch import EpBuffers, ep_dispatch
    torch.manual_seed(41)
    t, h, e, k = 77, 1024, 16, 4
    x = torch.randn(t, h, device=DEV, dtype=torch.bfloat16)
    logits = torch.randn(t, e, device=DEV)
    w, ids = torch.topk(torch.softmax(logits, -1), k)
    ids = ids.to(torch.int32)
    ids[5, 1] = -1                                   # an inactive slot
    dev = torch.device("cuda", 0)
    plain = EpBuffers(_solo_group(), dev, e, h, 128, k)
    quant = EpBuffers(_solo_group(), dev, e, h, 128, k, fp8_dispatch=True)
    rows, offs, _ = ep_dispatch(None, x, ids, w.float(), e, plain)
    (rq, rs), offs_q, _ = ep_dispatch(None, x, ids, w.float(), e, quant, fp8=True)
    torch.cuda.synchronize()
    n = int(offs[-1])
    assert n == t * k - 1 and torch.equal(offs, offs_q)
    # rows of one expert arrive in an order fixed by atomics: compare expert by expert as multisets
    want_q, want_s = ops.quant_fp8_1x128(rows[:n].contiguous())
    for ei in range(e):
        lo, hi = int(offs[ei]), int(offs[ei + 1])
        a = torch.cat([want_q[lo:hi].view(torch.uint8).float(), want_s[lo:hi]], dim=1)
        b = torch.cat([rq[lo:hi].view(torch.uint8).float(), rs[lo:hi]], dim=1)
        assert torch.equal(torch.sort(a, dim=0).values, torch.sort(b, dim=0).values)
    plain.close(), quant.close()
    ops.check_status()


@pytest.mark.parametrize("sink_len,window", [(4, 8), (0, 6), (3, 0)])
def test_sink_window_latent_attention_cuda_matches_the_cpu_path(sink_len, window):
    """Learned sink rows + sliding window on the latent cache, as composed on the GPU (sparse mode of
    the latent-cache kernel with its log-sum-exp, the sink GEMM, the LSE merge kernel), against the
    fp32 CPU path of the same module with the same weights."""
    from omni_npu_b200.attention.metadata import AttentionMetadata, set_forward_context
    from omni_npu_b200.attention.mla import MLABackend, StaticSinkMLAAttention
    from omni_npu_b200.config import ModelConfig
    from omni_npu_b200.models.utils import random_init_
    kw = dict(architecture="DeepseekV3ForCausalLM", model_type="deepseek_v3", hidden_size=512, num_layers=1,
              num_heads=16, num_kv_heads=16, head_dim=192, intermediate_size=1024, vocab_size=512,
              rms_norm_eps=1e-6, rope_theta=10000.0, max_position_embeddings=512, rope_neox=False,
              use_mla=True, q_lora_rank=0, kv_lora_rank=512, qk_nope_head_dim=128, qk_rope_head_dim=64,
              v_head_dim=128)
    dev = torch.device("cuda", 0)
    gpu = StaticSinkMLAAttention(ModelConfig(dtype=torch.bfloat16, **kw), 0, dev, "model.layers.0.self_attn",
                                 sink_len=sink_len, sliding_window=window)
    random_init_(gpu, seed=3, std=0.05)
    if sink_len:
        gpu.param_sink_kv.data.normal_(0, 0.5)
    cpu = StaticSinkMLAAttention(ModelConfig(dtype=torch.float32, **kw), 0, torch.device("cpu"),
                                 "model.layers.0.self_attn", sink_len=sink_len, sliding_window=window)
    cpu.load_state_dict({k: v.float().cpu() for k, v in gpu.state_dict().items()})
    gpu.process_weights_after_loading(), cpu.process_weights_after_loading()
    bs, nblk, lens = 16, 8, [21, 13]
    T = sum(lens)
    torch.manual_seed(1)
    hidden = (torch.randn(T, 512) * 0.5).to(torch.bfloat16)
    pos = torch.cat([torch.arange(n) for n in lens]).to(torch.int32)
    bt = torch.tensor([[1, 2, 0, 0], [3, 4, 0, 0]], dtype=torch.int32)
    slots = torch.cat([bt[b, torch.arange(n) // bs] * bs + torch.arange(n) % bs for b, n in enumerate(lens)]).to(torch.int32)
    cu = torch.tensor([0, lens[0], T], dtype=torch.int32)
    outs = {}
    for name, mod, d, dt in (("gpu", gpu, dev, torch.bfloat16), ("cpu", cpu, torch.device("cpu"), torch.float32)):
        cache = MLABackend.allocate_kv_cache(nblk, bs, 512, 64, dt, d)
        md = AttentionMetadata(is_prefill=True, num_seqs=2, num_tokens=T, max_q_len=max(lens), max_seq_len=max(lens),
                               q_len=0, positions=pos.to(d), slot_mapping=slots.to(d), block_tables=bt.to(d),
                               seq_lens=torch.tensor(lens, dtype=torch.int32, device=d), cu_q=cu.to(d),
                               num_actual_tokens=T, num_actual_seqs=2)
        with set_forward_context(md, [cache]):
            outs[name] = mod(hidden.to(d, dt)).float().cpu()
    got, want = outs["gpu"], outs["cpu"]
    rel = (got - want).abs().max() / want.abs().max().clamp_min(1e-6)
    assert rel <= 5e-2, float(rel)
    ops.check_status()
