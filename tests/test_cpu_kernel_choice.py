"""What the layers tell the kernels, and which kernel a call takes: rules on the host, checked without a GPU."""
import pytest
import torch

from omni_npu_b200 import ops
from omni_npu_b200.layers.linear import Fp8BlockLinearMethod, UnquantizedLinearMethod
from omni_npu_b200.layers.norm import RMSNorm
from omni_npu_b200.layers.quant_fp8 import fp8_block_gemm, quantize_weight_block


def _record(monkeypatch, name):
    calls, real = [], getattr(ops, name)

    def wrapped(*a, **k):
        calls.append(k)
        return real(*a, **k)

    monkeypatch.setattr(ops, name, wrapped)
    return calls


def test_only_parameters_are_read_ahead_of_the_kernels_before(monkeypatch):
    """A product may load its weights early only where the caller says that no kernel writes them: a layer's parameters,
    not the expanded copy of e4m3 weights that is made right ahead of the product."""
    calls = _record(monkeypatch, "gemm")
    x, layer = torch.randn(3, 64), torch.nn.Module()
    layer.weight = torch.nn.Parameter(torch.randn(32, 64), requires_grad=False)
    UnquantizedLinearMethod().apply(layer, x, None)
    assert calls.pop()["w_ready"] is True
    wq, ws = quantize_weight_block(torch.randn(32, 64))
    layer.weight, layer.weight_scale_inv = (torch.nn.Parameter(t, requires_grad=False) for t in (wq, ws))
    Fp8BlockLinearMethod().apply(layer, x, None)
    fp8_block_gemm(x, wq, ws, w_ready=True)
    assert len(calls) == 2 and not any(c.get("w_ready", False) for c in calls)


def test_norm_layers_read_their_parameters_early(monkeypatch):
    norm, x = RMSNorm(16, dtype=torch.float32), torch.randn(2, 16)
    alone, added = _record(monkeypatch, "rms_norm"), _record(monkeypatch, "fused_add_rms_norm")
    norm(x), norm(x, x.clone())
    assert alone.pop()["w_ready"] is True and added.pop()["w_ready"] is True
    ops.rms_norm(x, norm.weight.data, 1e-6)
    assert not alone.pop().get("w_ready", False)


def _qwen_attention():
    """One attention layer of a small Qwen3 model, and what it returns for a prompt of five tokens."""
    from omni_npu_b200.attention.metadata import AttentionMetadata, set_forward_context
    from omni_npu_b200.config import ModelConfig
    from omni_npu_b200.engine.llm import build_engine_config
    from omni_npu_b200.models.llama import LlamaAttention
    from omni_npu_b200.worker.worker import Worker
    mc = ModelConfig(hidden_size=64, num_layers=1, num_heads=4, num_kv_heads=2, head_dim=16, intermediate_size=64,
                     vocab_size=64, max_position_embeddings=64, qk_norm=True, dtype=torch.float32)
    cfg = build_engine_config(mc, device="cpu", max_num_seqs=1, num_gpu_blocks=4, block_size=16)
    Worker(cfg, local_rank=0, rank=0).init_device()
    torch.manual_seed(0)
    attn = LlamaAttention(mc, 0, "cpu", "attn")
    for p in attn.parameters():
        p.data.normal_(0.0, 0.2)
    i32 = dict(dtype=torch.int32)
    md = AttentionMetadata(is_prefill=True, num_seqs=1, num_tokens=5, max_q_len=5, max_seq_len=5, q_len=0,
                           positions=torch.arange(5, **i32), slot_mapping=torch.arange(5, **i32),
                           block_tables=torch.zeros(1, 1, **i32), seq_lens=torch.tensor([5], **i32),
                           cu_q=torch.tensor([0, 5], **i32), num_actual_tokens=5, num_actual_seqs=1)
    x = torch.randn(5, 64)

    def run():
        caches = [tuple(torch.zeros(4, 2, 16, 16) for _ in range(2))]
        with set_forward_context(md, caches, cfg):
            return attn(x)

    return attn, run


def test_head_norms_that_somebody_watches_are_called(monkeypatch):
    """Hooks on the head norms, wrapped classes (the name-list tracer's) and modules of other classes see their calls."""
    attn, run = _qwen_attention()
    want, seen = run(), []
    handle = attn.k_norm.register_forward_hook(lambda m, a, out: seen.append("hook"))
    torch.testing.assert_close(run(), want)
    handle.remove()
    real = RMSNorm.forward
    monkeypatch.setattr(RMSNorm, "forward", lambda self, *a, **k: (seen.append("class"), real(self, *a, **k))[1])
    torch.testing.assert_close(run(), want)
    monkeypatch.undo()
    assert seen == ["hook", "class", "class"]

    class Doubled(RMSNorm):
        def forward(self, x):
            return 2 * super().forward(x)

    plain = attn.q_norm
    attn.q_norm = Doubled(16, plain.eps, torch.float32)
    attn.q_norm.weight.data.copy_(plain.weight)
    doubled = run()
    attn.q_norm = plain
    plain.weight.data.mul_(2)
    torch.testing.assert_close(doubled, run())


def test_head_norms_keep_an_eps_of_their_own():
    attn, run = _qwen_attention()
    attn.q_norm.eps, attn.k_norm.eps = 1e-6, 10.0
    got = run()
    norms = [m.eps for m in (attn.q_norm, attn.k_norm)]
    handle = attn.q_norm.register_forward_hook(lambda *a: None)         # the modules are called one by one
    want = run()
    handle.remove()
    torch.testing.assert_close(got, want)
    attn.k_norm.eps = 1e-6
    assert norms == [1e-6, 10.0] and (run() - got).abs().max() > 1e-3


@pytest.mark.parametrize("n,k", [(128, 4096), (4096, 4096), (4096, 7168), (4700, 4096), (9216, 4096), (9000, 4096),
                                 (18944, 2048), (130, 256), (640, 64)])
def test_split_products_keep_within_a_limit_of_ctas(n, k):
    """A product that shares K among CTAs uses no more of them than its caller allows, and all of K's slabs."""
    splits = ops._core().gemm_stream_splits
    tiles, slabs = -(-n // 128), -(-k // 64)
    for limit in (0, 1, 8, 32, 64, 100, 148, 296, 1000):
        s = splits(n, k, limit, 148)
        assert s in (1, 2, 4, 8) and (s == 1 or tiles * s <= min(limit or 296, 296))
        assert s == 1 or ((s - 1) * -(-slabs // s) < slabs and -(-slabs // s) >= 4)
        assert s <= splits(n, k, 0, 148)
        assert tiles * s <= {1: tiles, 2: 296, 4: 284, 8: 264}[s]          # clusters that are resident at once


@pytest.mark.parametrize("quant", [None, "fp8"])
def test_experts_choose_kernels_by_the_rows_of_the_step(monkeypatch, quant):
    """Not by the size of the receive buffer, which on several ranks holds the largest step."""
    from types import SimpleNamespace

    from omni_npu_b200.layers import moe
    from omni_npu_b200.layers.moe_dispatch import DispatchHandle
    h, experts, cap = 128, 2, 4096
    buffers = SimpleNamespace(fp8_dispatch=False, expert_y=torch.zeros(cap, h))
    layer = SimpleNamespace(ep_size=1, buffers=buffers, shared_experts=None, quant=quant, num_physical=experts,
                            intermediate_size=h, act=ops.SILU, unary=None, w13=torch.randn(experts, 2 * h, h),
                            w2=torch.randn(experts, h, h), w13_scale=torch.ones(experts, 2, 1),
                            w2_scale=torch.ones(experts, 1, 1))
    layer._expert_rows = lambda *a, **k: moe.FusedMoE._expert_rows(layer, *a, **k)
    handle = DispatchHandle(None, None, None, 5, cap, None, expected_rows=10)
    monkeypatch.setattr(moe, "ep_dispatch", lambda *a, **k: (torch.zeros(cap, h), torch.tensor([0, 4, 10]), handle))
    monkeypatch.setattr(moe, "ep_combine", lambda comm, y, *a: y)
    seen = []
    for name in ("grouped_gemm", "grouped_gemm_fp8_block"):
        monkeypatch.setattr(ops, name, lambda a, *p, **k: (seen.append(k.get("rows")), torch.zeros(cap, h))[1])
    moe.FusedMoE._routed(layer, SimpleNamespace(is_cuda=True, device=None), None, None)
    assert seen == [10, 10]


def test_rows_of_a_step_choose_the_grouped_kernel():
    few, many = ops.grouped_rows_tile(16, 16, 1536), ops.grouped_rows_tile(131072, 16, 1536)
    assert few > 0 and many == 0            # streamed weights; CTA pairs
    # a single tile of weight rows per group: never pairs; a long K with some rows: the kernel with rows of A as M
    assert [ops.grouped_rows_tile(16 * r, 16, 128, 512) for r in (16, 512, 768, 1024, 2048)] == [32, 32, 64, 64, 128]
    assert [ops.grouped_rows_tile(8 * r, 8, 128, 2048) for r in (16, 17, 4096)] == [32, -1, -1]


def test_rows_that_stream_their_weights():
    """Split products up to 128 rows whatever their width; others where the kernel is the fastest of equal ones."""
    assert ops.stream_parts(4096, 4096) > 1 and ops.stream_rows(4096, 4096) == 128
    assert ops.stream_parts(12288, 4096) == 1 and ops.stream_rows(12288, 4096) == 16
    assert ops.stream_rows(12288, 4096, 0, False) == 128            # without the CTA-pair kernel
    assert ops.stream_parts(2048, 512) == 1 and ops.stream_rows(2048, 512) == 63
    assert ops.stream_rows(128256, 4096) == ops.stream_rows(32, 256) == 128
    assert ops.stream_rows(4096, 4096, 8) == 63                     # a limit of CTAs leaves no split


@pytest.mark.parametrize("items", [1, 8, 100, 148, 149, 2048])
@pytest.mark.parametrize("keys", [1, 255, 256, 511, 512, 2300, 8192, 163840])
def test_latent_splits_leave_keys_for_each(items, keys):
    s = ops.latent_splits(items, keys)
    assert 1 <= s <= 16 and (s == 1 or keys // s >= 256)
    if items >= 148 * 16 or keys < 512:
        assert s == 1
    if items == 1 and keys >= 16 * 256:
        assert s > 1
