"""Kernels that exist in several forms, chosen by size: every form against float64 at the sizes where it can go
wrong, and, in the 32-bit path, the same bits from each of them."""
import math

import numpy as np
import pytest
import torch

from test_kernels_gpu import DEV, _attention_reference, _ops, _paged_case, _rand

pytestmark = pytest.mark.gpu


# -- 32-bit products -----------------------------------------------------------------------------
ROWS, ROWS_WIDE, TILE, PAIR, PAIR_WIDE, FEW, BLOCK = 1, 2, 3, 4, 5, 6, 7


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (8, 9, 60), (9, 2305, 68), (16, 8193, 36), (3, 8200, 68), (8, 8200, 100), (12, 4700, 68),
                                   (16, 10300, 36), (24, 8200, 36), (64, 65, 772), (65, 63, 128),
                                   (129, 200, 1028), (200, 130, 16)])
def test_gemm_simt_forms_give_the_same_bits(M, N, K):
    """Remainders of rows, features and k in every form, and the sizes at which the rule takes each of the few-row forms; the
    residual form; strided rows.  Error: K roundings of 2^-24 of sums that stay below sum |a w|, a random walk of them."""
    from sglang_c_b200.csrc import build
    ops, lib = _ops(), build.load("gemm_simt")
    wide = _rand(M, K + 12, seed=M)
    a, w, bias = wide[:, 4:4 + K], _rand(N, K, seed=N), _rand(N, seed=K)
    ref = a.double() @ w.double().t() + bias.double()
    first = None
    try:
        for form in (ROWS, ROWS_WIDE, TILE, PAIR, PAIR_WIDE, FEW, BLOCK, 0):
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
    bound = float((a.double().abs() @ w.double().abs().t() + bias.double().abs()).max()) * 2.0 ** -24 * (K + 1) ** 0.5
    assert float((first.double() - ref).abs().max()) < bound


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


@pytest.mark.parametrize("H,Hkv,D,ps,window", [(16, 4, 64, 16, None), (16, 16, 128, 8, 40), (30, 2, 36, 16, 33), (30, 30, 4, 32, None)])
def test_attention_f32_portions_have_the_general_kernels_bits(H, Hkv, D, ps, window):
    """Portions of several requests in blocks of 32 tokens, against the kernel of a token a warp and float64: prompts and a
    portion behind a context, lengths off the edges of tiles and blocks."""
    ops = _ops()
    lens, q_lens = [330, 97, 333], [330, 97, 63] if D >= 64 else [330, 97, 133]
    c = _paged_case(lens, q_lens, H, Hkv, D, ps, torch.float32, seed=D)
    T, scale, outs = sum(q_lens), 1.3 / math.sqrt(D), []
    assert ops.attention_f32_form(T, H, D, 330, 3) == "portions" and ops.attention_f32_form(T, H, D, 330, 0) == "general"
    for n_portions in (0, 3):
        out = torch.full((T, H * D), float("nan"), device=DEV)
        ops.attention_simt(c["q"], c["cache"], c["bt"], c["token_req"], c["positions"], out, H, scale, window, 333, max_q_len=330,
                           n_portions=n_portions)
        outs.append(out)
    assert torch.equal(*outs)
    assert float((outs[0].double().cpu() - _attention_reference(c, H, Hkv, D, scale, window)).abs().max()) < 2e-5


@pytest.mark.parametrize("D,at", [(64, 9), (64, 61), (128, 40)])
def test_attention_f32_keeps_a_bad_value_from_the_tokens_before_it(D, at):
    """A value that is infinite or no number reaches the tokens that see it, and no other token of its tile or block."""
    ops = _ops()
    H, ps, lens, q_lens = 8, 16, [70, 640], [70, 600]
    c = _paged_case(lens, q_lens, H, H, D, ps, torch.float32, seed=at)
    T = sum(q_lens)

    def run():
        out = torch.zeros(T, H * D, device=DEV)
        ops.attention_simt(c["q"], c["cache"], c["bt"], c["token_req"], c["positions"], out, H, 0.1, None, 640, max_q_len=600, n_portions=2)
        return out

    assert ops.attention_f32_form(T, H, D, 600, 2) == "portions"

    clean = run()
    for bad in (float("inf"), float("nan")):
        key = 40 + at                                   # (the second request's token `at`: its first token is at position 40)
        c["cache"][int(c["bt"][1, key // ps]), 1, :, key % ps] = bad
        out = run()
        assert torch.equal(out[:70 + at], clean[:70 + at])
        assert not bool(torch.isfinite(out[70 + at:]).any())


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


@pytest.mark.parametrize("H,Hkv,D", [(40, 1, 64), (20, 2, 128)])
def test_prompt_attention_of_many_query_tiles(H, Hkv, D):
    """More query tiles than half of the blocks that run at once: tiles of five key tiles are split, shorter ones are not."""
    ops = _ops()
    lens, q_lens, ps = [600, 129, 40, 700], [130, 129, 40, 200], 16
    c = _paged_case(lens, q_lens, H, Hkv, D, ps, torch.bfloat16, seed=H)
    q_start = torch.tensor(np.concatenate([[0], np.cumsum(q_lens)]), dtype=torch.int32, device=DEV)
    kv_len = torch.tensor(lens, dtype=torch.int32, device=DEV)
    out = torch.full((sum(q_lens), H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
    scale = 1.0 / math.sqrt(D)
    ops.attention_prefill_tc(c["q"], c["cache"], c["bt"], q_start, kv_len, out, H, scale, None, len(lens), max(q_lens))
    # bfloat16 weights and results of size below one: 2^-8 each
    assert float((out.double().cpu() - _attention_reference(c, H, Hkv, D, scale, None)).abs().max()) < 1.2e-2


@pytest.mark.parametrize("kv_shared", [False, True])
@pytest.mark.parametrize("q_lens", [[1, 1, 1, 44], [70, 1, 1, 1, 1], [1] * 33 + [129] + [1] * 3, [1] * 40 + [2], [3] + [1] * 31 + [5] + [1] * 31 + [140],
                                    [1, 9, 1, 9]])
def test_a_launch_for_the_portions_alone(q_lens, kv_shared):
    """The number of single tokens is known: portions first, last, beyond the 32nd and the 64th request and between single
    tokens are all found, and no single token's row is written."""
    ops = _ops()
    H, D, ps = 3, 64, 16
    lens = [n + (37 * r) % 150 for r, n in enumerate(q_lens)]
    c = _paged_case(lens, q_lens, H, 1, D, ps, torch.bfloat16, seed=len(q_lens))
    if kv_shared:                                       # (rows that are keys and values at once)
        c["cache"], c["Vs"] = c["cache"][:, :1].contiguous(), c["Ks"]
    starts = np.concatenate([[0], np.cumsum(q_lens)])
    q_start = torch.tensor(starts, dtype=torch.int32, device=DEV)
    kv_len = torch.tensor(lens, dtype=torch.int32, device=DEV)
    out = torch.full((sum(q_lens), H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
    singles = [int(s) for s, n in zip(starts, q_lens) if n == 1]
    ops.attention_prefill_tc(c["q"], c["cache"], c["bt"], q_start, kv_len, out, H, 0.1, None, len(lens), max(q_lens), skip_single=len(singles),
                             kv_shared=kv_shared)
    rows = torch.ones(sum(q_lens), dtype=torch.bool)
    rows[singles] = False
    assert bool(torch.isnan(out[~rows]).all())
    ref = _attention_reference(c, H, 1, D, 0.1, None)
    assert float((out.double().cpu() - ref)[rows].abs().max()) < 2e-2


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


@pytest.mark.parametrize("T", [9, 18, 40])
def test_decode_attention_keeps_a_bad_key_in_every_share(T):
    """A key that is no number, near the front of a request's keys, in the middle or near their end: the request's result
    is none either, whichever block has that key; the other requests' results keep their bits."""
    ops = _ops()
    H, D, ps = 12, 64, 16
    lens = [650 + r for r in range(T)]
    c = _paged_case(lens, [1] * T, H, H, D, ps, torch.bfloat16, seed=T)

    def run(cache):
        out = torch.zeros(T, H * D, dtype=torch.bfloat16, device=DEV)
        ops.attention_decode(c["q"], cache, c["bt"], None, c["positions"], out, H, 0.1, None, max(lens), variant="stream", n_tokens=T)
        return out

    clean = run(c["cache"])
    for key in (3, 200, 340, 500, 640):
        cache = c["cache"].clone()
        cache[int(c["bt"][1, key // ps]), 0, :, key % ps] = float("nan")
        out = run(cache)
        assert bool(torch.isnan(out[1]).all()), key
        assert torch.equal(torch.cat([out[:1], out[2:]]), torch.cat([clean[:1], clean[2:]])), key


# -- recurrences in chunks ----------------------------------------------------------------------------
def _walk(mode, q, k, v, gates, decay, H, G, D, V, S):
    n = q.shape[0]
    q, k, v = (t.double().reshape(n, -1, w) for t, w in ((q, D), (k, D), (v, V)))
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    out = torch.zeros(n, H, V, dtype=torch.float64, device=DEV)
    for t in range(n):
        S = S * (gates[t, H:] if mode == "delta" else decay).double()[:, None, None]
        u = gates[t, :H].double()[:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])) if mode == "delta" else v[t]
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return out.reshape(n, H * V), S


@pytest.mark.parametrize("silu", [False, True])
@pytest.mark.parametrize("mode,H,G,D,V,rate", [("delta", 4, 2, 64, 64, 0.1), ("delta", 3, 3, 40, 100, 0.002), ("delta", 2, 1, 7, 9, 3.0),
                                               ("decay", 2, 2, 64, 64, 0.05), ("decay", 2, 2, 33, 70, 0.5)])
def test_recurrences_in_chunks(mode, H, G, D, V, rate, silu):
    """Portions of 1 to 200 tokens over shuffled slots: chunk edges, states carried in, decays near one, far from it
    and zero, sizes no vector load fits, silu of the inputs.  The chunks may not be further off than 2 x the walk token by
    token."""
    ops = _ops()
    g = torch.Generator().manual_seed(D)
    lens = [200, 1, 64, 65, 127]
    T, R = sum(lens), len(lens)
    q, k, v = (torch.randn(T, n, generator=g).to(DEV) for n in (G * D, G * D, H * V))
    k = torch.nn.functional.normalize(k.reshape(T, G, D), dim=-1).reshape(T, G * D).contiguous()
    gates = torch.cat([torch.rand(T, H, generator=g), torch.exp(-rate * 2 * torch.rand(T, H, generator=g))], 1).to(DEV)
    if rate > 1:
        gates[::19, H:] = 0.0
    decay = torch.exp(-rate * torch.arange(1, H + 1)).to(DEV)
    S0 = torch.randn(R + 2, H, D, V, generator=g).to(DEV)
    starts, slots = np.concatenate([[0], np.cumsum(lens)]), [3, 0, 6, 1, 4]
    i32 = lambda x: torch.tensor(np.asarray(x), dtype=torch.int32, device=DEV)      # noqa: E731
    kw = dict(gates=gates, silu_in=silu) if mode == "delta" else dict(head_decay=decay, silu_in=silu)
    act = (lambda x: torch.nn.functional.silu(x.double())) if silu else (lambda x: x)
    got = {}
    for way in ("walk", "chunks"):
        S, o = S0.clone(), torch.full((T, H * V), float("nan"), device=DEV)
        if way == "walk":
            ops.matrix_state(mode, q, k, v, o, S, i32(starts), i32(slots), R, H, G, D, V, **kw)
        else:
            ws = torch.full((ops.delta_chunks_workspace(mode, T, R, H, V),), float("nan"), device=DEV)
            ops.delta_chunks(mode, q, k, v, o, S, i32(starts), i32(slots), R, H, G, D, V, ws, **kw)
        got[way] = (o, S)
    for r, slot in enumerate(slots):
        at = slice(starts[r], starts[r + 1])
        want, state = _walk(mode, act(q[at]), act(k[at]), act(v[at]), gates[at], decay, H, G, D, V, S0[slot].double())
        for i, (ref, pick) in enumerate(((want, lambda t: t[0][at]), (state, lambda t: t[1][slot]))):
            err = {w: float((pick(got[w]).double() - ref).norm() / ref.norm()) for w in got}
            assert err["chunks"] < max(2.0 * err["walk"], 5e-7), (r, i, err)
    for slot in set(range(R + 2)) - set(slots):
        assert torch.equal(got["chunks"][1][slot], S0[slot])


@pytest.mark.parametrize("mode", ["delta", "decay"])
@pytest.mark.parametrize("at,what", [(5, "v"), (13, "k"), (62, "v"), (71, "q"), (90, "gates")])
def test_chunks_keep_a_bad_number_from_the_tokens_before_it(mode, at, what):
    """An infinity or NaN of one token: the tokens before it and the other requests keep their bits, as they do where
    the recurrence goes token by token."""
    ops = _ops()
    g = torch.Generator().manual_seed(at)
    H, G, D, V, lens = 2, 1, 64, 70, [100, 130]
    T, R = sum(lens), len(lens)
    x = {n: torch.randn(T, w, generator=g).to(DEV) for n, w in (("q", G * D), ("k", G * D), ("v", H * V))}
    x["k"] = torch.nn.functional.normalize(x["k"], dim=-1)
    x["gates"] = torch.rand(T, 2 * H, generator=g).to(DEV)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)      # noqa: E731
    kw = dict(gates=x["gates"]) if mode == "delta" else dict(head_decay=torch.rand(H, generator=g).to(DEV))
    outs = []
    for bad in (None, float("inf"), float("nan")):
        if bad is not None:
            x[what][lens[0] + at] = bad
        o, S = torch.zeros(T, H * V, device=DEV), torch.zeros(R, H, D, V, device=DEV)
        ws = torch.empty(ops.delta_chunks_workspace(mode, T, R, H, V), device=DEV)
        ops.delta_chunks(mode, x["q"], x["k"], x["v"], o, S, i32([0, lens[0], T]), i32([1, 0]), R, H, G, D, V, ws, **kw)
        outs.append((o, S))
    for o, S in outs[1:]:
        assert torch.equal(o[:lens[0] + at], outs[0][0][:lens[0] + at]) and torch.equal(S[1], outs[0][1][1])


# -- steps of one token a request ------------------------------------------------------------------------
@pytest.mark.parametrize("mode,H,G,D,V", [("delta", 4, 2, 64, 64), ("delta", 3, 3, 40, 100), ("delta", 2, 1, 129, 68), ("delta", 2, 2, 256, 4),
                                          ("decay", 3, 3, 64, 64), ("decay", 2, 2, 7, 12), ("decay", 2, 2, 128, 132)])
def test_recurrences_of_single_tokens(mode, H, G, D, V):
    """Key sizes at the edges of the rows a thread keeps, value sizes of one tile, a part of one and several; no further
    off than 2 x the walk, or a handful of roundings."""
    ops = _ops()
    g = torch.Generator().manual_seed(D + V)
    R = 5
    q, k, v = (torch.randn(R, n, generator=g).to(DEV) for n in (G * D, G * D, H * V))
    k = torch.nn.functional.normalize(k.reshape(R, G, D), dim=-1).reshape(R, G * D).contiguous()
    gates = torch.rand(R, 2 * H, generator=g).to(DEV)
    decay = torch.rand(H, generator=g).to(DEV)
    S0 = torch.randn(R + 2, H, D, V, generator=g).to(DEV)
    slots = [3, 0, 6, 1, 4]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)      # noqa: E731
    kw = dict(gates=gates) if mode == "delta" else dict(head_decay=decay)
    for silu in (False, True):
        got = {}
        for way in ("walk", "step"):
            S, o = S0.clone(), torch.full((R, H * V), float("nan"), device=DEV)
            if way == "walk":
                ops.matrix_state(mode, q, k, v, o, S, i32(list(range(R + 1))), i32(slots), R, H, G, D, V, silu_in=silu, **kw)
            else:
                ops.delta_step(mode, q, k, v, o, S, i32(slots), H, G, D, V, silu_in=silu, **kw)
            got[way] = (o, S)
        act = (lambda t: torch.nn.functional.silu(t.double())) if silu else (lambda t: t)
        for r, slot in enumerate(slots):
            at = slice(r, r + 1)
            want, state = _walk(mode, act(q[at]), act(k[at]), act(v[at]), gates[at], decay, H, G, D, V, S0[slot].double())
            for ref, pick in ((want, lambda t: t[0][at]), (state, lambda t: t[1][slot])):
                err = {w: float((pick(got[w]).double() - ref).norm() / ref.norm()) for w in got}
                assert err["step"] < max(2.0 * err["walk"], 5e-7), (silu, r, err)
        for slot in set(range(R + 2)) - set(slots):
            assert torch.equal(got["step"][1][slot], S0[slot])


@pytest.mark.parametrize("taps,D,V", [(2, 12, 7), (3, 33, 64), (4, 64, 32)])
def test_short_convolution_of_single_tokens(taps, D, V):
    """Token by token or as one portion: the same bits, and the same inputs left for the next step."""
    ops = _ops()
    g = torch.Generator().manual_seed(taps)
    R, n, G, H = 3, 6, 2, 3
    C = 2 * G * D + H * V
    x = torch.randn(n, R, C + 2 * H, generator=g).to(DEV)
    w, a_log, dt = torch.randn(C, taps, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV)
    segs = [(0, G, D, 1, D ** -0.5), (G * D, G, D, 1, 1.0), (2 * G * D, H, V, 0, 1.0)]
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)      # noqa: E731
    tail0 = torch.randn(5, taps - 1, C, generator=g).to(DEV)

    def run(rows, lens, tail):
        T = sum(lens)
        y, gates = torch.empty(T, C, device=DEV), torch.empty(T, 2 * H, device=DEV)
        starts = np.concatenate([[0], np.cumsum(lens)]).tolist()
        ops.short_conv(rows.contiguous(), w, tail, y, i32([r for r, m in enumerate(lens) for _ in range(m)]), i32(starts), i32([3, 1, 4]),
                       R, segs, gates=(H, C, C + H, a_log, dt, gates))
        return y, gates

    whole, stepped = tail0.clone(), tail0.clone()
    y, gates = run(x.transpose(0, 1).reshape(R * n, -1), [n] * R, whole)
    steps = [run(x[t], [1] * R, stepped) for t in range(n)]
    assert torch.equal(y.view(R, n, C).transpose(0, 1), torch.stack([s[0] for s in steps]))
    assert torch.equal(gates.view(R, n, -1).transpose(0, 1), torch.stack([s[1] for s in steps]))
    assert torch.equal(whole, stepped)


@pytest.mark.parametrize("taps,D,V", [(2, 12, 7), (3, 33, 64), (4, 64, 32)])
def test_short_convolution_of_long_portions(taps, D, V):
    """Portions long enough to go by runs of tokens, and the same in pieces that do not: the same bits, and the same inputs
    left for the next step; a portion that starts inside a run, one of three tokens, tails of an earlier step."""
    ops = _ops()
    g = torch.Generator().manual_seed(10 + taps)
    lens, G, H, slots = [700, 3, 598], 4, 9, [3, 1, 4]
    T, R, C = sum(lens), len(lens), 2 * G * D + H * V
    x = torch.randn(T, C + 2 * H, generator=g).to(DEV)
    w, a_log, dt = torch.randn(C, taps, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV)
    segs = [(0, G, D, 1, D ** -0.5), (G * D, G, D, 1, 1.0), (2 * G * D, H, V, 0, 1.0)]
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)      # noqa: E731
    tail0, starts = torch.randn(5, taps - 1, C, generator=g).to(DEV), np.concatenate([[0], np.cumsum(lens)]).tolist()

    def run(rows, tail, lens, slots):
        y, gates = torch.empty(sum(lens), C, device=DEV), torch.empty(sum(lens), 2 * H, device=DEV)
        ops.short_conv(rows.contiguous(), w, tail, y, i32([r for r, m in enumerate(lens) for _ in range(m)]),
                       i32(np.concatenate([[0], np.cumsum(lens)]).tolist()), i32(slots), len(lens), segs, gates=(H, C, C + H, a_log, dt, gates))
        return torch.cat([y, gates], 1)

    whole, pieces = tail0.clone(), tail0.clone()
    got = run(x, whole, lens, slots)
    cut = [run(x[s + p:s + min(p + 61, n)], pieces, [min(61, n - p)], [slot]) for s, n, slot in zip(starts, lens, slots) for p in range(0, n, 61)]
    assert torch.equal(got, torch.cat(cut)) and torch.equal(whole, pieces)


@pytest.mark.parametrize("E,top", [(1, 1), (8, 8), (8, 3), (31, 5), (32, 32), (33, 4), (96, 8)])
def test_router_order_of_choice(E, top):
    """Logits with many ties on both sides of 32 experts: the larger first, the lower index first among equals."""
    ops = _ops()
    T = 37
    z = torch.randint(-3, 4, (T, E), generator=torch.Generator().manual_seed(E), dtype=torch.int64).float().to(DEV)
    dense, ids, wts = torch.empty(T, E, device=DEV), torch.empty(T, top, dtype=torch.int32, device=DEV), torch.empty(T, top, device=DEV)
    ops.router(z, None, dense, ids, wts, top, renorm=True, weight_scale=1.5)
    want = torch.sort(z, dim=1, descending=True, stable=True).indices[:, :top]
    assert torch.equal(ids.long(), want)
    s = torch.sigmoid(z.double())
    w = torch.gather(s, 1, want)
    w = w / w.sum(1, keepdim=True) * 1.5
    assert float((wts.double() - w).abs().max()) < 1e-6
    assert float((dense.double() - torch.zeros_like(s).scatter(1, want, w)).abs().max()) < 1e-6


@pytest.mark.parametrize("width", [64, 65, 256, 257])
def test_gated_norm_at_the_edges_of_what_a_lane_keeps(width):
    ops = _ops()
    g = torch.Generator().manual_seed(width)
    T, groups = 5, 3
    o, z = (torch.randn(T, groups * width, generator=g).to(DEV) for _ in range(2))
    gain = torch.randn(width, generator=g).to(DEV)
    x = o.double().view(T, groups, width)
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * gain.double()
    for act, gate in (("silu", torch.nn.functional.silu(z.double())), ("sigmoid", torch.sigmoid(z.double())), ("none", None)):
        y = torch.empty_like(o)
        ops.gated_norm(o, None if gate is None else z, gain, y, groups, width, 1e-5, act)
        want = x.reshape(T, -1) * (1.0 if gate is None else gate)
        # about ten 32-bit roundings a value (2^-24 each) and a sum of `width` squares
        assert float(((y.double() - want).abs() / (want.abs() + 1e-3)).max()) < 1e-5


def test_cache_writing_projection_over_a_long_k():
    """Sizes whose plain product is dealt over K: the projection that writes the cache is still taken, and right."""
    ops = _ops()
    M, H, Hkv, D, K, ps = 200, 6, 1, 64, 2304, 16
    N, n_pages = (H + 2 * Hkv) * D, 13
    assert ops.gemm_tc_form(M, N, K) == "few"
    g = torch.Generator().manual_seed(K)
    a, w = (torch.randn(n, K, generator=g).mul_(s).to(DEV, torch.bfloat16) for n, s in ((M, 1.0), (N, 0.02)))
    slots = torch.randperm(n_pages * ps, generator=g)[:M].to(DEV, torch.int32)
    out = torch.zeros(M, N, dtype=torch.bfloat16, device=DEV)
    cache = torch.zeros(n_pages, 2, Hkv, ps, D, dtype=torch.bfloat16, device=DEV)
    assert ops.gemm_tc_kv(a, w, None, out, cache, slots, H, Hkv, D)
    want = a.double() @ w.double().T
    got = torch.cat([out[:, :H * D].double()] + [cache[slots.long() // ps, i, 0, slots.long() % ps].double() for i in range(2)], 1)
    # half a unit of bfloat16 a value and the 32-bit sums before it
    assert float((got - want).abs().max()) < float(want.abs().max()) * 2.0 ** -8


@pytest.mark.parametrize("M,N,K,shares", [(129, 768, 3072, 8), (170, 768, 3104, 7), (160, 1000, 3072, 6), (250, 768, 3072, 5), (320, 700, 4096, 4),
                                          (400, 768, 3080, 3), (129, 2048, 2120, 3), (768, 768, 3072, 2), (4700, 60, 2304, 2)])
def test_many_tokens_over_a_long_k(M, N, K, shares):
    """K dealt to two to eight blocks, tokens off the edges of tiles of 32, features off those of 128."""
    ops = _ops()
    assert ops.gemm_tc_shares(M, N, K) == shares
    g = torch.Generator().manual_seed(M)
    a, w = (torch.randn(n, K, generator=g).mul_(s).to(DEV, torch.bfloat16) for n, s in ((M, 1.0), (N, 0.02)))
    bias, x = torch.randn(N, generator=g).to(DEV), torch.randn(M, N, generator=g).to(DEV)
    plain = a.double() @ w.double().T + bias.double()
    want = x.double() + plain
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.gemm_tc(a, w, bias, out=out)
    ops.gemm_tc(a, w, bias, residual=x)
    # 32-bit sums of K products: K roundings of 2^-24 of sums that stay below sum |a w|, a random walk of them
    bound = float((a.double().abs() @ w.double().abs().T).max()) * 2.0 ** -24 * K ** 0.5
    assert float((x.double() - want).abs().max()) < bound
    assert float((out.double() - plain).abs().max()) < float(plain.abs().max()) * 2.0 ** -8      # half a unit of bfloat16


@pytest.mark.parametrize("M,N,K", [(1, 128, 3072), (16, 1152, 4608), (5, 100, 3080), (16, 768, 8200), (17, 768, 3072), (16, 1160, 3072)])
def test_few_tokens_over_a_long_k(M, N, K):
    """K dealt to more than eight blocks, evenly and not, and the sizes just beyond."""
    ops = _ops()
    g = torch.Generator().manual_seed(K + M)
    a, w = (torch.randn(n, K, generator=g).mul_(s).to(DEV, torch.bfloat16) for n, s in ((M, 1.0), (N, 0.02)))
    bias, x = torch.randn(N, generator=g).to(DEV), torch.randn(M, N, generator=g).to(DEV)
    want = x.double() + a.double() @ w.double().T + bias.double()
    ops.gemm_tc(a, w, bias, residual=x)
    # 32-bit sums of K products: K roundings of 2^-24 of sums that stay below sum |a w|, a random walk of them
    bound = float((a.double().abs() @ w.double().abs().T).max()) * 2.0 ** -24 * K ** 0.5
    assert float((x.double() - want).abs().max()) < bound


@pytest.mark.parametrize("M,N,K", [(45, 2304, 768), (64, 768, 768), (56, 16400, 128), (65, 1000, 776), (128, 1030, 1024), (97, 1600, 1608),
                                   (33, 130, 3080), (70, 770, 3072), (13, 4800, 1600), (24, 100, 64)])
def test_few_tokens_in_tiles_of_16_and_32(M, N, K):
    """Tokens, features and K off the tiles' edges, K whole and in two to eight shares, more blocks than are resident at once."""
    ops = _ops()
    assert ops.gemm_tc_form(M, N, K) == "few"
    a, w, bias, x = _rand(M, K, dtype=torch.bfloat16, seed=1), _rand(N, K, dtype=torch.bfloat16, seed=2), _rand(N, seed=3), _rand(M, N, seed=4)
    plain = a.double() @ w.double().t() + bias.double()
    want = x.double() + plain
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.gemm_tc(a, w, bias, out=out)
    ops.gemm_tc(a, w, bias, residual=x)
    # 32-bit sums of K products: K roundings of 2^-24 of sums that stay below sum |a w|, a random walk of them
    bound = float((a.double().abs() @ w.double().abs().t()).max()) * 2.0 ** -24 * K ** 0.5 + 1e-5
    assert float((x.double() - want).abs().max()) < bound
    assert float((out.double() - plain).abs().max()) < float(plain.abs().max()) * 2.0 ** -8      # half a unit of bfloat16


@pytest.mark.parametrize("rows,E,form,gain,bias", [(1024, 768, "rms", True, False), (1025, 8, "layer", True, True), (1031, 1600, "rms", False, False),
                                                   (1500, 2048, "layer", True, False), (1024, 132, "rms", True, True), (1023, 768, "rms", True, False)])
def test_norms_of_many_rows(rows, E, form, gain, bias):
    """A warp a row from 1,024 rows on: widths that end inside a warp's pieces, a gather, a strided source and destination."""
    ops = _ops()
    wide = _rand(rows, E + 12, seed=E)
    x = wide[:, 4:4 + E]
    g, b = (_rand(E, seed=1) if gain else None), (_rand(E, seed=2) if bias else None)
    pick = torch.randperm(rows, generator=torch.Generator().manual_seed(3)).to(torch.int32).to(DEV)
    for rows_of in (None, pick):
        out = torch.full((rows, E + 8), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.norm_rows(x, g, b, 1e-5, out[:, :E], form, src_rows=rows_of)
        d = x.double() if rows_of is None else x.double()[rows_of.long()]
        d = d - d.mean(-1, keepdim=True) if form == "layer" else d
        want = d / torch.sqrt((d * d).mean(-1, keepdim=True) + 1e-5)
        want = want * (1.0 if g is None else g.double()) + (0.0 if b is None else b.double())
        # half a unit of bfloat16, and the 32-bit roundings before it
        assert float(((out[:, :E].double() - want).abs() - want.abs() * 2.0 ** -8).max()) < 1e-5
        assert bool(torch.isnan(out[:, E:]).all())


@pytest.mark.parametrize("T,groups,act", [(683, 12, "silu"), (2051, 4, "sigmoid"), (8195, 1, "none"), (682, 12, "silu")])
def test_gated_norm_of_many_rows_of_64(T, groups, act):
    """Sixteen lanes a row from 8,192 rows on: a number of rows that leaves warps in part, a gain for all rows and one each."""
    ops = _ops()
    o, z = _rand(T, groups * 64 + 8, seed=T)[:, :groups * 64], _rand(T, groups * 64, seed=4)
    for gains in (64, groups * 64):
        gain = _rand(gains, seed=5)
        y = torch.empty(T, groups * 64, dtype=torch.bfloat16, device=DEV)
        ops.gated_norm(o, None if act == "none" else z, gain, y, groups, 64, 1e-5, act)
        x = o.double().reshape(T, groups, 64)
        x = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * gain.double().reshape(-1, 64)).reshape(T, -1)
        s = torch.sigmoid(z.double())
        want = x * {"none": 1.0, "sigmoid": s, "silu": s * z.double()}[act]
        assert float(((y.double() - want).abs() - want.abs() * 2.0 ** -8).max()) < 1e-5


@pytest.mark.parametrize("rows,F,per,act", [(3, 8, 8, "silu"), (700, 264, 24, "silu"), (2049, 1024, 128, "silu"), (65, 80, 16, "gelu_tanh"), (300, 4096, 0, "silu")])
def test_gated_activations_in_16_byte_pieces(rows, F, per, act):
    """A piece, two pieces and a remainder a thread; weights of blocks of columns, some zero; large and very negative gates."""
    ops = _ops()
    src = _rand(rows, 2 * F, dtype=torch.bfloat16, seed=F, scale=4.0)
    src[0, :4] = torch.tensor([90.0, -90.0, 3.0e4, -3.0e4], device=DEV)
    w = None
    if per:
        w = torch.rand(rows, F // per, generator=torch.Generator().manual_seed(1)).to(DEV)
        w[::3, 0] = 0.0
    dst = torch.full((rows, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.gated_act(src, dst, weights=w, per=per, act=act)
    g, u = src[:, :F].double(), src[:, F:].double()
    want = (g * torch.sigmoid(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * u
    if per:
        want = want * w.double().repeat_interleave(per, 1)
    # half a unit of bfloat16, and a few 2^-22 of the fast exponential and division (times the gate's size in the exponent)
    assert float(((dst.double() - want).abs() - want.abs() * (2.0 ** -8)).max()) < 1e-4


def test_gated_activations_skip_what_was_not_chosen():
    """Columns of weight zero are not read: 2 of 8 experts take a quarter of the reads of 8 of 8 (in bytes 0.5 of the
    time with the stores; the bound leaves room for the clock), and what they hold does not matter."""
    ops = _ops()
    rows, X, per = 2048, 8, 1024
    srcs = [_rand(rows, 2 * X * per, dtype=torch.bfloat16, seed=i) for i in range(3)]          # 67 MB each: beyond the L2 together
    dst = torch.empty(rows, X * per, dtype=torch.bfloat16, device=DEV)
    pick = torch.rand(rows, X, generator=torch.Generator().manual_seed(1)).argsort(1)[:, :2]
    few, all_ = torch.zeros(rows, X).scatter(1, pick, 0.5).to(DEV), torch.full((rows, X), 0.5, device=DEV)

    def us(w):
        best = 1e9
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for s in srcs * 4:
                ops.gated_act(s, dst, weights=w, per=per)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert us(few) < 0.75 * us(all_)
    clean = dst.clone()
    ops.gated_act(srcs[0], clean, weights=few, per=per)
    hole = (few == 0).repeat_interleave(per, 1)
    ops.gated_act(torch.where(torch.cat([hole, hole], 1), torch.full_like(srcs[0], float("nan")), srcs[0]), dst, weights=few, per=per)
    assert torch.equal(dst, clean) and bool((dst[hole] == 0).all())


@pytest.mark.parametrize("rows", [(1 << 30) - 1, (1 << 30) + 5])
def test_gated_activations_of_a_billion_pieces(rows):
    """The counters of 32 and of 64 bits on both sides of 2^30 pieces: one piece a row, all rows alike (17 GB of results)."""
    ops = _ops()
    one = _rand(1, 16, dtype=torch.bfloat16, seed=1)
    dst = torch.empty(rows, 8, dtype=torch.bfloat16, device=DEV)
    for act in ("silu", "gelu_tanh"):
        for w in (None, torch.full((1, 1), 0.5, device=DEV)):
            dst.fill_(float("nan"))
            want = torch.empty(1, 8, dtype=torch.bfloat16, device=DEV)
            ops.gated_act(one, want, weights=w, per=8, act=act)
            ops.gated_act(one.expand(rows, 16), dst, weights=None if w is None else w.expand(rows, 1), per=8, act=act)
            for part in dst.view(torch.int64).split(1 << 28):
                assert bool((part == want.view(torch.int64)).all())


@pytest.mark.parametrize("E,groups,form", [(4, 1, "rms"), (512, 1, "layer"), (128, 6, "rms"), (1028, 1, "layer"), (2044, 1, "rms"), (2048, 2, "layer"),
                                           (4096, 1, "rms"), (4100, 1, "layer")])
def test_norms_of_a_few_rows(E, groups, form):
    """Up to two 16-byte pieces a thread, and a row beyond: with a gather, skipped rows, and added to what is there."""
    ops = _ops()
    n, W = 5, E * groups
    x, g, b, there = _rand(n, W + 4, seed=E)[:, :W], _rand(W, seed=1), _rand(W, seed=2), _rand(n + 2, W, seed=3)
    pick, place = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ((4, 0, 3, 3, 1), (2, 6, -1, 0, 5)))
    d = x.double().view(n, groups, E)
    d = d - d.mean(-1, keepdim=True) if form == "layer" else d
    want = (d / torch.sqrt((d * d).mean(-1, keepdim=True) + 1e-5)).view(n, W) * g.double() + b.double()
    tol = 1e-5      # a sum of up to 4,100 squares in 32-bit and a handful of roundings of values below 20
    got = torch.empty(n, W, device=DEV)
    ops.norm_rows(x, g, b, 1e-5, got, form, src_rows=pick, groups=groups)
    assert float((got.double() - want[pick.long()]).abs().max()) < tol
    added = there.clone()
    ops.norm_rows(x, g, b, 1e-5, added, form, add=True, dst_rows=place, groups=groups)
    sure = there.double()
    for r, p in enumerate(place.tolist()):
        if p >= 0:
            sure[p] += want[r]
    assert float((added.double() - sure).abs().max()) < tol
    assert torch.equal(added[[1, 3, 4]], there[[1, 3, 4]])
    half = torch.empty(n, W, dtype=torch.bfloat16, device=DEV)
    ops.norm_rows(x, None, None, 1e-5, half, form, groups=groups)
    plain = (d / torch.sqrt((d * d).mean(-1, keepdim=True) + 1e-5)).view(n, W)
    assert float(((half.double() - plain).abs() - plain.abs() * 2.0 ** -8).max()) < tol


@pytest.mark.parametrize("E,K,T", [(1, 8, 3), (8, 768, 8), (17, 1024, 148), (33, 1032, 5), (40, 264, 149), (9, 769, 4)])
def test_router_makes_its_logits(E, K, T):
    """Rows that a lane keeps whole and longer ones, more experts than warps, tokens on both sides of the SMs."""
    ops = _ops()
    h, w = _rand(T, K, seed=K).bfloat16(), (_rand(E, K, seed=E) / K ** 0.5).bfloat16()
    top = min(E, 3)
    dense, ids, wts = torch.empty(T, E, device=DEV), torch.empty(T, top, dtype=torch.int32, device=DEV), torch.empty(T, top, device=DEV)
    ops.router(None, None, dense, ids, wts, top, rows=h, matrix=w)
    s = torch.sigmoid(h.double() @ w.double().t())
    best = torch.topk(s, top, dim=1)
    # a logit's error is below 2^-24 times the sum of its products' sizes times the additions a lane makes; near ties may fall either way
    assert float((wts.double() - best.values).abs().max()) < 1e-5
    assert float((dense.gather(1, ids.long()).double() - torch.gather(s, 1, ids.long())).abs().max()) < 1e-5


@pytest.mark.parametrize("E,K", [(1, 520), (8, 769), (32, 64), (33, 769), (40, 520)])
def test_router_makes_its_logits_in_32_bits(E, K):
    """The 32-bit product: the end of a row inside the loads on their way at once; and a token's weights have the same bits in
    a launch of 149 tokens, which share SMs, as in launches of a few."""
    ops = _ops()
    T, top = 149, min(E, 3)
    h, w = _rand(T, K + 4, seed=K)[:, :K], _rand(E, K, seed=E) / K ** 0.5

    def run(lo, hi):
        n = hi - lo
        dense, ids, wts = torch.empty(n, E, device=DEV), torch.empty(n, top, dtype=torch.int32, device=DEV), torch.empty(n, top, device=DEV)
        ops.router(None, None, dense, ids, wts, top, rows=h[lo:hi], matrix=w)
        return dense, ids, wts

    whole = run(0, T)
    parts = [run(lo, hi) for lo, hi in ((0, 1), (1, 9), (9, T))]
    for i in range(3):
        assert torch.equal(whole[i], torch.cat([p[i] for p in parts]))
    s = torch.sigmoid(h.double() @ w.double().t())
    best = torch.topk(s, top, dim=1)
    # a lane adds up to 25 products and the warp 5 times, 2^-24 of sums below 4 each; a near tie may fall either way
    assert float((whole[2].double() - best.values).abs().max()) < 4 * 30 * 2.0 ** -24
    assert float((whole[0].gather(1, whole[1].long()).double() - torch.gather(s, 1, whole[1].long())).abs().max()) < 4 * 30 * 2.0 ** -24


@pytest.mark.parametrize("D,V,splits", [(64, 64, 2), (64, 40, 8), (128, 72, 9), (256, 256, 11)])
def test_merge_of_a_tokens_shares(D, V, splits):
    """Shares on both sides of the eight that are fetched at once, values that end inside a warp, gates of both kinds and a sink."""
    ops = _ops()
    T, H, G, ps, n = 3, 6, 2, 16, 380
    pages = (n + ps - 1) // ps
    cache = _rand(pages, G * ps * (D + V), seed=D).bfloat16()
    q = _rand(T, H * D, seed=V).bfloat16()
    table = torch.arange(pages, dtype=torch.int32, device=DEV).repeat(T, 1)
    req, pos = torch.arange(T, dtype=torch.int32, device=DEV), torch.tensor([n - 1, 40, 0], dtype=torch.int32, device=DEV)
    for sinks, gate in ((None, None), (_rand(H, seed=5), _rand(T, H, seed=6)), (None, _rand(T, H * V, seed=7))):
        def run(s, **more):
            out = torch.empty(T, H * V, dtype=torch.bfloat16, device=DEV)
            ops.attention_ext(q, cache, table, req, pos, out, H, G, D, V, ps, D ** -0.5, None, None, sinks, n, gate=gate, splits=s, **more)
            return out.double()
        one = run(1)
        dealt = run(splits, max_q_len=1, workspace=torch.empty(T * H * splits * (V + 2), device=DEV))
        # both round a 32-bit result to bfloat16 once: a unit of it apart at most
        assert float(((dealt - one).abs() - one.abs() * 2.0 ** -7).max()) < 1e-5


def test_rotary_rows_have_the_same_bits_beside_many_and_few_tokens():
    """A warp a row for few tokens, four warps for many; heads wider than what a lane has on its way at once."""
    ops = _ops()
    T, H, G, D, V, ps, dims = 150, 7, 2, 272, 40, 16, 96
    x = _rand(T, H * D + G * (D + V), seed=1)
    pos, freq = torch.arange(T, dtype=torch.int32, device=DEV) * 7, torch.logspace(0, -4, dims // 2, dtype=torch.float64, device=DEV)
    def run(lo, hi, q, cache):
        ops.rotary_kv(x[lo:hi], pos[lo:hi], freq, 1.25, dims, 1e-6, q[lo:hi], cache, torch.arange(lo, hi, dtype=torch.int32, device=DEV), H, G, D, V, ps)
    made = []
    for cuts in (((0, T),), ((0, 1), (1, 20), (20, T))):
        q, cache = torch.zeros(T, H * D, device=DEV), torch.zeros((T + ps - 1) // ps, G * ps * (D + V), device=DEV)
        for lo, hi in cuts:
            run(lo, hi, q, cache)
        made.append((q, cache))
    assert torch.equal(made[0][0], made[1][0]) and torch.equal(made[0][1], made[1][1])
    head = x[:, :D].double()
    a = pos.double()[:, None] * freq
    u, v = head[:, :dims // 2], head[:, dims // 2:dims]
    turned = torch.cat([(u * a.cos() - v * a.sin()) * 1.25, (v * a.cos() + u * a.sin()) * 1.25, head[:, dims:]], 1)
    want = turned / torch.sqrt((turned * turned).mean(-1, keepdim=True) + 1e-6)
    # the angle is rounded to 32 bits inside one turn: 2^-24 * 2 pi, and a few roundings of values below 6
    assert float((made[0][0][:, :D].double() - want).abs().max()) < 1e-5


@pytest.mark.parametrize("T", [1, 148, 149])
def test_rotary_rounds_as_it_is_written(T):
    """u cos - v sin and u sin + v cos with the first product inside the multiply-add and the second one rounded, in each
    form of the kernel (cosines and sines by turning rows of ones and zeros)."""
    ops = _ops()
    H, G, D, ps, dims = 5, 2, 64, 16, 48
    half, width = dims // 2, (H + G) * D + G * D
    pos, freq = torch.arange(T, dtype=torch.int32, device=DEV) * 7 + 1, torch.logspace(0, -4, half, dtype=torch.float64, device=DEV)

    def run(x):
        q, cache = torch.zeros(T, H * D, device=DEV), torch.zeros((T + ps - 1) // ps, G * ps * 2 * D, device=DEV)
        ops.rotary_kv(x, pos, freq, 1.0, dims, None, q, cache, torch.arange(T, dtype=torch.int32, device=DEV), H, G, D, D, ps)
        return q.view(T, H, D)

    unit = torch.zeros(T, width, device=DEV)
    unit.view(T, -1, D)[:, :, :half] = 1.0
    turn = run(unit).double()
    cs, sn = turn[..., :half], turn[..., half:dims]
    x = _rand(T, width, seed=T)
    rows = x.view(T, -1, D)[:, :H].double()
    u, v = rows[..., :half], rows[..., half:dims]
    got, once = run(x), lambda z: z.float().double()          # (a product of two 32-bit numbers is exact in 64 bits)
    assert torch.equal(got[..., :half], (u * cs - once(v * sn)).float())
    assert torch.equal(got[..., half:dims], (u * sn + once(v * cs)).float())


@pytest.mark.parametrize("E", [4, 1020, 1024, 1028, 1664, 1668, 4096])
def test_layer_norm_at_the_edges_of_a_blocks_warps(E):
    """Blocks of up to 8, 13 and 32 warps, whose partial sums are added in one order: the same bits in both precisions' rounding."""
    ops = _ops()
    x, g, b = _rand(5, E, seed=E) + 3.0, _rand(E, seed=1), _rand(E, seed=2)
    out, half = torch.empty(5, E, device=DEV), torch.empty(5, E, dtype=torch.bfloat16, device=DEV)
    ops.layernorm(x, g, b, 1e-5, out)
    ops.layernorm(x, g, b, 1e-5, half)
    assert torch.equal(out.bfloat16(), half)
    want = torch.nn.functional.layer_norm(x.double(), (E,), g.double(), b.double(), 1e-5)
    # sums of up to 4,096 numbers in 32-bit: an error of some 2^-24 * 12 of the mean of 3, times a gain below 5 and 1 / deviation (4 numbers: below 10)
    assert float((out.double() - want).abs().max()) < 1e-4
