"""Rules by which launches choose a kernel or a split, at the sizes that they were measured at (no GPU)."""
from types import SimpleNamespace

import pytest
import torch

from sglang_c_b200.csrc import ops
from sglang_c_b200.engine.runtime import Runtime


@pytest.mark.parametrize("keys,blocks,width,splits", [
    (64, 24, 128, 1), (128, 24, 128, 5), (256, 24, 128, 9), (512, 24, 128, 16), (1024, 24, 128, 16), (100, 96, 128, 4),
    (512, 48, 128, 8), (256, 64, 128, 4), (100, 128, 128, 2), (512, 32, 48, 8), (2000, 48, 128, 9), (128, 384, 128, 1),
    (100, 16, 256, 5), (512, 16, 256, 8), (256, 32, 256, 4), (100, 64, 256, 2)])
def test_a_tile_a_share_only_where_every_tile_has_one(keys, blocks, width, splits):
    assert ops.attention_ext_splits(keys, None, None, blocks, width) == splits
    assert ops.attention_ext_splits(4 * keys, keys, None, blocks, width) == splits          # (a window)
    assert ops.attention_ext_splits(4 * keys, None, keys, blocks, width) == splits          # (a chunk)


@pytest.mark.parametrize("tokens,heads,dim,longest,portions,form", [
    (128, 12, 64, 128, 1, "general"), (384, 12, 64, 384, 1, "general"), (512, 12, 64, 512, 1, "portions"), (256, 25, 64, 256, 1, "portions"),
    (512, 8, 128, 512, 1, "general"), (640, 8, 128, 640, 1, "portions"), (512, 12, 64, 16, 32, "general"), (512, 12, 64, 32, 16, "portions"),
    (32, 12, 64, 2, 16, "general"), (512, 12, 64, 481, 0, "general"), (1000, 12, 32, 1000, 1, "portions"), (960, 12, 32, 120, 8, "general"),
    (512, 12, 66, 512, 1, "general"), (512, 12, 132, 512, 1, "general"), (1 << 22, 1, 64, 1 << 22, 1, "general"),
    (8, 12, 64, 1, 0, "singles"), (24, 12, 64, 1, 0, "singles"), (32, 12, 64, 1, 0, "general"), (64, 12, 64, 1, 0, "singles"),
    (128, 12, 64, 1, 0, "general"), (256, 12, 64, 1, 0, "general"), (16, 8, 128, 1, 0, "singles"), (24, 8, 128, 1, 0, "general"),
    (64, 8, 128, 1, 0, "general"), (256, 12, 32, 1, 0, "singles")])
def test_32_bit_attention_takes_the_kernel_that_was_faster(tokens, heads, dim, longest, portions, form):
    assert ops.attention_f32_form(tokens, heads, dim, longest, portions) == form


@pytest.mark.parametrize("singles", [0, 1, 31])
def test_a_step_with_single_tokens_is_no_step_of_portions(monkeypatch, singles):
    """What the runtime tells the 32-bit kernels of a step: single tokens beside portions would take turns with them."""
    told = []
    monkeypatch.setattr(ops, "attention_simt", lambda *a, n_portions=0, **kw: told.append(n_portions))
    rt = Runtime.__new__(Runtime)
    rt.dtype = "float32"
    q = torch.zeros(4, 8)
    ctx = SimpleNamespace(n_decode=singles, R=2 + singles, max_q_len=9, token_req=None, positions=None, max_keys=9)
    grp, binding = SimpleNamespace(block_table=None, slots=None), SimpleNamespace(tensor=torch.zeros(1, 2, 1, 4, 8), write=False)
    rt.attend(ctx, q, q, q, binding, grp, q, 1, 1, 8, 1.0, None)
    rt.attend_shared(ctx, q, binding, grp, q, 1, 8, 1.0, None)
    assert told == ([0, 0] if singles else [2, 2])


@pytest.mark.parametrize("M,N,K,shares", [(1, 768, 3072, 16), (16, 768, 3072, 16), (17, 768, 3072, 8), (16, 768, 3008, 8), (16, 1024, 3072, 8),
                                          (16, 1024, 3584, 14), (16, 1152, 4608, 15), (16, 1160, 4608, 8), (8, 128, 8200, 15)])
def test_shares_of_a_long_k(M, N, K, shares):
    """Clusters of more than eight blocks only where the device holds them, and where they pay."""
    assert ops.gemm_tc_shares(M, N, K) == shares
    assert ops.gemm_tc_shares(M, N, K, 8) == 8


@pytest.mark.parametrize("M,N,K,shares", [(129, 768, 3072, 8), (256, 768, 3072, 5), (320, 768, 4096, 4), (400, 768, 3072, 3), (512, 768, 3072, 2),
                                          (256, 1024, 4096, 4), (768, 768, 3072, 2), (800, 768, 3072, 1), (129, 2048, 3072, 3), (512, 768, 2048, 1)])
def test_shares_of_many_tokens(M, N, K, shares):
    assert ops.gemm_tc_shares(M, N, K) == shares


# (walk and chunks measured, in us, beside each)
@pytest.mark.parametrize("mode,lens,heads,dim,v_dim,chunks", [
    ("delta", [150], 12, 64, 64, False),               # 35, 37
    ("delta", [200], 12, 64, 64, True),                # 45, 37
    ("delta", [512] * 4, 12, 64, 64, True),            # 158, 75
    ("delta", [200] * 8, 12, 64, 64, False),           # 72, 75
    ("delta", [1024] * 2, 12, 64, 64, True),           # 227, 80
    ("delta", [512] * 4, 16, 32, 32, False),           # 96, 100
    ("delta", [512] * 4, 32, 64, 128, False),          # 226, 320
    ("delta", [1024] * 2, 32, 64, 128, True),          # 418, 318
    ("delta", [200], 12, 65, 64, False),               # (no form in chunks)
    ("delta", [2] * 30 + [900], 12, 64, 64, False),    # (more requests than chunks)
    ("decay", [100], 3, 64, 64, False),                # 29, 28
    ("decay", [128], 3, 64, 64, True),                 # 34, 28
    ("decay", [134, 133, 133], 32, 64, 128, False),    # 63, 66
    ("decay", [200, 100, 100], 32, 64, 128, True),     # 87, 62
    ("decay", [128], 64, 64, 16, False),               # 34, 36
    ("decay", [512] * 4, 64, 64, 16, False),           # 176, 226
    ("decay", [100] * 8, 64, 64, 16, False),           # 55, 116
    ("decay", [1024] * 2, 3, 64, 64, True)])           # 229, 30
def test_recurrences_go_in_chunks_where_those_are_faster(mode, lens, heads, dim, v_dim, chunks):
    assert ops.delta_chunks_pay(mode, sum(lens), len(lens), max(lens), heads, dim, v_dim) == chunks
