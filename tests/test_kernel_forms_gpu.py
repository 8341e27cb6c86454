"""Kernels that exist in several forms, chosen by size: every form against float64 at the sizes where it can go
wrong, and, in the 32-bit path, the same bits from each of them."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, _ops, _rand

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
