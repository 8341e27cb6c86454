"""Which kernel, and how many blocks a (token, head) item, the decode attention takes: at the sizes it was measured at (no GPU)."""
import pytest

from sglang_c_b200.csrc import build


@pytest.mark.parametrize("T,H,max_keys,form", [
    (1, 12, 128, 1), (8, 12, 128, 1), (64, 12, 128, 1),                     # short contexts: no merge
    (8, 12, 640, 5), (8, 12, 1024, 4), (1, 12, 640, 8),                     # few items: all blocks resident at once
    (16, 12, 256, 1), (16, 12, 512, 2), (28, 12, 256, 1), (40, 12, 256, 1),
    (12, 12, 1024, 0), (28, 12, 512, 0), (64, 12, 512, 0), (64, 12, 1024, 0),       # 0: the streaming kernel
    (1, 1, 1024, 8), (7, 1, 2048, 8), (4, 1, 4096, 8), (1, 1, 8192, -1),            # very few items (-1: the older rule, 32 shares)
    (4, 12, 3200, 8), (5, 12, 2600, 8), (6, 12, 1300, 8), (8, 12, 2048, 8),         # long contexts in two or three rounds of blocks
    (8, 12, 4000, 0), (12, 12, 2048, 0), (13, 12, 1300, 0), (48, 12, 2048, 0)])
def test_decode_attention_takes_what_was_faster(T, H, max_keys, form):
    lib = build.load("attention_decode_tma")
    assert lib.sglc_attention_decode_form(T, H, 64, 16, max_keys, 0) == form


def test_decode_attention_forms_have_no_answer_for_other_sizes():
    lib = build.load("attention_decode_tma")
    for D, page in ((128, 16), (32, 16), (64, 128), (64, 0)):
        assert lib.sglc_attention_decode_form(8, 12, D, page, 512, 0) == -1
    assert lib.sglc_attention_decode_form(4000, 12, 64, 16, 1024, 0) == 0
    assert lib.sglc_attention_decode_form(4000, 12, 64, 3, 1024, 0) == -1    # (neither the streaming kernel nor the other takes it)
