"""The 32-bit products on the tensor cores: every form (tile of tokens, blocks that share a tile's K) against float64, with
the same bits from each of them."""
import pytest
import torch

from test_kernels_gpu import DEV, _ops, _rand

pytestmark = pytest.mark.gpu

FORMS = [(16, 1), (16, 3), (16, 16), (32, 1), (32, 8), (64, 1), (64, 12), (96, 1), (128, 1)]


def _lib():
    from sglang_c_b200.csrc import build
    return build.load("gemm_f32")


def _each(run):
    """run() once in every form that takes the sizes (a form whose blocks hold too many sums refuses), and as chosen."""
    ops, lib, out = _ops(), _lib(), []
    try:
        for form in FORMS + [(0, 0)]:
            lib.sglc_gemm_f32_set_form(*form)
            try:
                out.append(run(ops))
            except ops.KernelError as e:
                assert "not supported" in str(e) and form != (0, 0), form
    finally:
        lib.sglc_gemm_f32_set_form(0, 0)
    assert len(out) >= 8
    return out


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (15, 127, 60), (17, 129, 64), (33, 128, 68), (129, 300, 772), (200, 65, 1604), (9, 257, 3076),
                                   (97, 20000, 8)])
def test_gemm_f32_forms_give_the_same_bits(M, N, K):
    """Remainders of rows, features, k and chunks.  An output's error at most: 24 additions into a chunk's sum, which tensor memory
    cuts, so 2^-23 of the sum of the chunk's |a w| each; 2^-24 of the whole sum a chunk; 2^-21 of each product left out or cut.
    All outputs' together: 5e-7 of sqrt(sum (a w)^2), three times the most seen; without one of the six products of pieces
    it is 4e-6 and more."""
    wide = _rand(M, K + 12, seed=M)
    a, w, bias = wide[:, 4:4 + K], _rand(N, K, seed=N), _rand(N, seed=K)
    ref = a.double() @ w.double().t() + bias.double()

    def run(ops):
        out = torch.full((M + 1, N), float("nan"), device=DEV)
        ops.gemm_f32(a, w, bias, out=out)
        assert bool(torch.isnan(out[M]).all())
        res = torch.ones(M, N, device=DEV)
        ops.gemm_f32(a, w, bias, residual=res)
        assert torch.equal(res, 1.0 + out[:M])
        act = torch.empty(M, N, device=DEV)
        ops.gemm_f32(a, w, bias, out=act, act="gelu_tanh")
        return out[:M], act

    each = _each(run)
    for out, act in each[1:]:
        assert torch.equal(out, each[0][0]) and torch.equal(act, each[0][1])
    out, act = each[0]
    scale = a.double().abs() @ w.double().abs().t() + bias.double().abs()
    bound = scale * (24 * 2.0 ** -23 + ((K + 63) // 64) * 2.0 ** -24 + 2.0 ** -21)
    assert bool(((out.double() - ref).abs() < bound).all())
    assert bool(((act.double() - torch.nn.functional.gelu(ref, approximate="tanh")).abs() < 1.2 * bound + 1e-6).all())
    plain = torch.empty(M, N, device=DEV)
    _ops().gemm_f32(a, w, None, out=plain)
    size = (a.double() ** 2 @ (w.double() ** 2).t()).sum().sqrt()
    assert float((plain.double() - a.double() @ w.double().t()).norm() / size) < 5e-7


def test_gemm_f32_is_closer_than_a_chain_of_multiply_adds():
    ops = _ops()
    for K in (640, 768, 3072):
        a, w, out, chain = _rand(300, K, seed=1), _rand(500, K, seed=2), torch.empty(300, 500, device=DEV), torch.empty(300, 500, device=DEV)
        ref = a.double() @ w.double().t()
        ops.gemm_f32(a, w, None, out=out)
        ops.gemm_simt(a, w, None, out=chain)
        assert float((out - ref).norm()) < 0.5 * float((chain - ref).norm())


def test_gemm_f32_numbers_at_the_edges():
    """Infinities and NaN come out as a chain of multiply-adds gives them; very large numbers are kept, and subnormal ones as far
    as bfloat16 has pieces for them: a number's last piece is a multiple of its smallest, 2^-133."""
    a, w = _rand(40, 200, seed=3), _rand(150, 200, seed=4)
    a[3, 7], a[5, 9], a[20, 100] = float("inf"), float("nan"), -float("inf")
    w[11, 7], w[140, 199] = 0.0, float("inf")
    a[30] = 0.0
    a[30, 0], a[31], a[32, :] = 1e-40, 0.0, 0.0
    w[:, 0] = 1.0
    a[31, 1], a[32, 0] = 3e38, 3.4028234e38
    w[:, 1] = 0.5
    ops = _ops()
    chain = torch.empty(40, 150, device=DEV)
    ops.gemm_simt(a, w, None, out=chain)

    def run(ops):
        out = torch.empty(40, 150, device=DEV)
        ops.gemm_f32(a, w, None, out=out)
        return out

    each = _each(run)
    for out in each:
        assert torch.equal(torch.nan_to_num(out), torch.nan_to_num(each[0]))
        assert torch.equal(torch.isnan(out), torch.isnan(chain)) and torch.equal(torch.isinf(out), torch.isinf(chain))
        keep = torch.isfinite(chain) & (w[:, 199] != float("inf"))[None]
        assert torch.equal(torch.sign(out[torch.isinf(chain)]), torch.sign(chain[torch.isinf(chain)]))
        assert torch.allclose(out[keep], chain[keep], rtol=2e-6, atol=2e-5)
        for r in (30, 31, 32):
            assert torch.allclose(out[r, :140], chain[r, :140], rtol=1e-6, atol=2.0 ** -133), r


@pytest.mark.parametrize("M,K", [(37, 68), (3, 200), (130, 132)])
def test_gemm_f32_outputs_that_are_no_numbers_at_the_edges(M, K):
    """NaN and infinities in the last token, k and feature: what a chain of multiply-adds gives, and the other outputs unchanged."""
    a, w, ops = _rand(M, K, seed=5), _rand(131, K, seed=6), _ops()
    clean, chain = torch.empty(M, 131, device=DEV), torch.empty(M, 131, device=DEV)
    ops.gemm_f32(a, w, None, out=clean)
    a[M - 1, K - 1], a[0, 0], w[130, K - 2], w[129, 1], w[128, 5] = float("nan"), float("inf"), float("nan"), -float("inf"), 3e38
    ops.gemm_simt(a, w, None, out=chain)

    def run(ops):
        out = torch.full((M, 131), 5.0, device=DEV)
        ops.gemm_f32(a, w, None, out=out)
        return out

    for out in _each(run):
        assert torch.equal(torch.isnan(out), torch.isnan(chain)) and torch.equal(out[torch.isinf(chain)], chain[torch.isinf(chain)])
        assert torch.equal(out[1:M - 1, :128], clean[1:M - 1, :128])
        assert torch.allclose(out[1:M - 1, 128], chain[1:M - 1, 128], rtol=1e-5)


def test_gemm_f32_of_nan_takes_a_few_times_the_time_and_no_more():
    """A step whose values have become NaN still ends soon: a chain for each output took 256 times the product's time (now 5)."""
    a, w, out, ops = _rand(1872, 768, seed=1), _rand(768, 768, seed=2), torch.empty(1872, 768, device=DEV), _ops()

    def ms(x):
        best = 1e9
        for _ in range(5):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record()
            for _ in range(5):
                ops.gemm_f32(x, w, None, out=out)
            e.record()
            e.synchronize()
            best = min(best, s.elapsed_time(e))
        return best

    usual, nan = ms(a), ms(torch.full_like(a, float("nan")))
    assert bool(torch.isnan(out).all()) and nan < 30 * usual


def test_gemm_f32_in_clusters_beside_clusters_of_another_stream():
    """Blocks that share a tile's K (320 to 512 of an SM's 512 columns of tensor memory) while few-token bfloat16 products, whose
    blocks share K too, run in another stream: a block gives its columns back before it waits for its peers."""
    ops, lib = _ops(), _lib()
    a, w = _rand(64, 768, seed=1), _rand(768, 768, seed=2)
    b, v = _rand(8, 768, seed=3).bfloat16(), _rand(768, 768, seed=4).bfloat16()
    n = 200
    outs = [torch.empty(64, 768, device=DEV) for _ in range(n)]
    halves = [torch.empty(8, 768, dtype=torch.bfloat16, device=DEV) for _ in range(n)]
    want, half = torch.empty_like(outs[0]), torch.empty_like(halves[0])
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    try:
        for form in ((64, 6), (64, 12), (32, 8), (16, 6)):
            lib.sglc_gemm_f32_set_form(*form)
            try:
                ops.gemm_f32(a, w, None, out=want)
            except ops.KernelError:
                continue
            ops.gemm_tc(b, v, None, out=half)
            torch.cuda.synchronize()
            for i in range(n):
                with torch.cuda.stream(one):
                    ops.gemm_f32(a, w, None, out=outs[i])
                with torch.cuda.stream(two):
                    ops.gemm_tc(b, v, None, out=halves[i])
            torch.cuda.synchronize()
            assert all(torch.equal(o, want) for o in outs) and all(torch.equal(h, half) for h in halves)
    finally:
        lib.sglc_gemm_f32_set_form(0, 0)


@pytest.mark.parametrize("M,H,Hkv,D,page", [(1, 12, 12, 64, 16), (37, 10, 10, 64, 16), (300, 8, 2, 96, 8), (70, 11, 3, 60, 5)])
def test_gemm_f32_kv_writes_the_cache(M, H, Hkv, D, page):
    """Queries, keys and values have the bits of the plain product, wherever a tile of 128 columns is cut; slots may be negative."""
    K, N = 644, (H + 2 * Hkv) * D
    a, w, bias = _rand(M, K, seed=1), _rand(N, K, seed=2, scale=0.1), _rand(N, seed=3)
    n_pages = (M + page - 1) // page + 2
    slots = torch.randperm(n_pages * page, generator=torch.Generator().manual_seed(4))[:M].to(torch.int32)
    slots[M // 2] = -1 if M > 2 else slots[M // 2]
    dev_slots = slots.to(DEV)
    plain = torch.empty(M, N, device=DEV)
    _ops().gemm_f32(a, w, bias, out=plain)
    keys, values = plain[:, H * D:(H + Hkv) * D].reshape(M, Hkv, D), plain[:, (H + Hkv) * D:].reshape(M, Hkv, D)
    want = torch.full((n_pages, 2, Hkv, page, D), 7.0, device=DEV)
    for t, s in enumerate(slots.tolist()):
        if s >= 0:
            want[s // page, 0, :, s % page], want[s // page, 1, :, s % page] = keys[t], values[t]

    def run(ops):
        out, cache = torch.full((M, N), float("nan"), device=DEV), torch.full((n_pages, 2, Hkv, page, D), 7.0, device=DEV)
        assert ops.gemm_f32_kv(a, w, bias, out, cache, dev_slots, H, Hkv, D)
        return out, cache

    for out, cache in _each(run):
        assert torch.equal(out[:, :H * D], plain[:, :H * D]) and bool(torch.isnan(out[:, H * D:]).all())
        assert torch.equal(cache, want)
