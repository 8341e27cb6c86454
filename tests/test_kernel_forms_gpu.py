"""Kernels that exist in several forms, chosen by size: every form against float64 at the sizes where it can go
wrong, and, in the 32-bit path, the same bits from each of them."""
import math

import numpy as np
import pytest
import torch

from test_kernels_gpu import DEV, _attention_reference, _ops, _paged_case, _rand

pytestmark = pytest.mark.gpu


# -- 32-bit products -----------------------------------------------------------------------------
ROWS, ROWS_WIDE, TILE, PAIR, PAIR_WIDE = 1, 2, 3, 4, 5


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (8, 9, 60), (9, 2305, 68), (16, 8193, 36), (64, 65, 772), (65, 63, 128),
                                   (129, 200, 1028), (200, 130, 16)])
def test_gemm_simt_forms_give_the_same_bits(M, N, K):
    """Remainders of rows, features and k in every form; the residual form; strided rows.  Error: K roundings of
    a sum of about sqrt(K) in size, each half a unit: below 1e-7 K."""
    from sglang_c_b200.csrc import build
    ops, lib = _ops(), build.load("gemm_simt")
    wide = _rand(M, K + 12, seed=M)
    a, w, bias = wide[:, 4:4 + K], _rand(N, K, seed=N), _rand(N, seed=K)
    ref = a.double() @ w.double().t() + bias.double()
    first = None
    try:
        for form in (ROWS, ROWS_WIDE, TILE, PAIR, PAIR_WIDE, 0):
            lib.sglc_gemm_simt_set_form(form)
            out = torch.full((M, N), float("nan"), device=DEV)
            ops.gemm_simt(a, w, bias, out=out)
            res = torch.ones(M, N, device=DEV)
            ops.gemm_simt(a, w, bias, residual=res)
            assert torch.equal(res, 1.0 + out)
            first = out if first is None else first
            assert torch.equal(out, first), form
    finally:
        lib.sglc_gemm_simt_set_form(0)
    assert float((first.double() - ref).abs().max()) < 1e-7 * K * math.sqrt(K) + 1e-6


# -- 32-bit attention ------------------------------------------------------------------------------
@pytest.mark.parametrize("H,Hkv,D,ps,window", [(2, 1, 64, 16, None), (3, 3, 128, 8, 40), (2, 2, 36, 16, 33), (1, 1, 4, 32, None)])
def test_attention_f32_has_the_same_bits_in_every_cut(H, Hkv, D, ps, window):
    """A token's result is the same, bit for bit, as part of a long portion, of a short one that begins inside a
    tile, beside other requests, and as a single token: blocks of 32 tokens, tiles of 32 keys, rounds of two."""
    ops = _ops()
    lens = [130, 31, 64, 1, 97]
    c = _paged_case(lens, lens, H, Hkv, D, ps, torch.float32, seed=D)
    T, starts, scale = c["q"].shape[0], np.concatenate([[0], np.cumsum(lens)]), 1.3 / math.sqrt(D)
    whole = torch.full((T, H * D), float("nan"), device=DEV)
    ops.attention_simt(c["q"], c["cache"], c["bt"], c["token_req"], c["positions"], whole, H, scale, window, max(lens), max_q_len=130)
    assert float((whole.double().cpu() - _attention_reference(c, H, Hkv, D, scale, window)).abs().max()) < 2e-5
    some = torch.tensor(sorted({int(s + i) for s, n in zip(starts, lens) for i in (0, 1, 30, 31, 32, 63, 64, 65, 95, 96, 129) if i < n}),
                        device=DEV)
    for pick, longest in ((some, 1), (some, 2), (torch.arange(33, 130, device=DEV), 97), (torch.arange(T - 97, T, device=DEV), 97)):
        out = torch.full((len(pick), H * D), float("nan"), device=DEV)
        ops.attention_simt(c["q"][pick].contiguous(), c["cache"], c["bt"], c["token_req"][pick].contiguous(),
                           c["positions"][pick].contiguous(), out, H, scale, window, max(lens), max_q_len=longest)
        assert torch.equal(out, whole[pick]), longest


# -- tensor-core prompt attention ---------------------------------------------------------------------
@pytest.mark.parametrize("D,window,grow", [(64, None, 3.0), (64, 150, 3.0), (128, None, 3.0), (64, None, 0.0), (64, None, -3.0)])
def test_prompt_attention_follows_a_growing_maximum(D, window, grow):
    """Scores whose maximum grows (or shrinks) by far more than 2^8 from key tile to key tile, so that the sums in
    tensor memory are scaled down again and again; ragged prompts, one behind a cached context.  bfloat16
    weights and results: 2^-8 of values of size about 3."""
    ops = _ops()
    H, Hkv, ps = 2, 1, 16
    lens, q_lens = [600, 129, 40], [470, 129, 40]
    c = _paged_case(lens, q_lens, H, Hkv, D, ps, torch.bfloat16, seed=D)
    one = torch.zeros(D)
    one[0] = 1.0
    for r, n in enumerate(lens):                      # the first entry of key p: grow * p / 16; of every query: 8
        c["Ks"][r][:, :, 0] = (grow * torch.arange(n)[:, None] / 16.0).to(torch.bfloat16)
        c["Qs"][r][:, :, 0] = 8.0
        for p in range(n):
            c["cache"][int(c["bt"][r, p // ps]), 0, :, p % ps] = c["Ks"][r][p].to(DEV)
    q = torch.cat([x.reshape(x.shape[0], H * D) for x in c["Qs"]]).to(DEV)
    T, scale = q.shape[0], 0.25
    q_start = torch.tensor(np.concatenate([[0], np.cumsum(q_lens)]), dtype=torch.int32, device=DEV)
    kv_len = torch.tensor(lens, dtype=torch.int32, device=DEV)
    out = torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.attention_prefill_tc(q, c["cache"], c["bt"], q_start, kv_len, out, H, scale, window, len(lens), max(q_lens))
    ref = _attention_reference(c, H, Hkv, D, scale, window)
    assert float((out.double().cpu() - ref).abs().max()) < 2.5e-2


# -- single tokens: items shared by clusters -------------------------------------------------------------
@pytest.mark.parametrize("T,H,Hkv,D,window", [(9, 12, 12, 64, None), (13, 16, 4, 64, None), (18, 12, 12, 64, 200), (6, 16, 16, 128, None),
                                              (3, 16, 2, 64, None)])
def test_stream_decode_shares_items_between_blocks(T, H, Hkv, D, window):
    """Contexts from one key to many tiles, so that ranks have full, short and empty runs of keys; the token's own
    key and value fused in.  bfloat16 results of size below 1: 2^-8."""
    ops = _ops()
    ps = 16
    lens = [int(n) for n in np.linspace(1, 700, T)]
    c = _paged_case(lens, [1] * T, H, Hkv, D, ps, torch.bfloat16, seed=T)
    scale = 0.9 / math.sqrt(D)
    ref = _attention_reference(c, H, Hkv, D, scale, window)
    k_new = torch.cat([K[-1:].reshape(1, Hkv * D) for K in c["Ks"]]).to(DEV)
    v_new = torch.cat([V[-1:].reshape(1, Hkv * D) for V in c["Vs"]]).to(DEV)
    both = torch.cat([k_new, v_new], 1).contiguous()
    slots = torch.tensor([int(c["bt"][r, (n - 1) // ps]) * ps + (n - 1) % ps for r, n in enumerate(lens)], dtype=torch.int32, device=DEV)
    for fused in (False, True):
        cache = c["cache"].clone()
        if fused:
            for r, n in enumerate(lens):
                cache[int(c["bt"][r, (n - 1) // ps]), :, :, (n - 1) % ps] = 0.0
        kw = dict(k_new=both[:, :Hkv * D], v_new=both[:, Hkv * D:], slots=slots) if fused else {}
        out = torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.attention_decode(c["q"], cache, c["bt"], None, c["positions"], out, H, scale, window, max(lens), variant="stream", n_tokens=T, **kw)
        assert float((out.double().cpu() - ref).abs().max()) < 1.2e-2, fused
        assert not fused or torch.equal(cache, c["cache"])
