"""What captured step graphs are told apart by (no GPU): steps that share a key take the same launches."""
from types import SimpleNamespace

import pytest

from buborax_models import BUB_B
from sglang_c_b200.config import resolve_architecture
from sglang_c_b200.engine.engine import Engine
from sglang_c_b200.engine.model import Model
from zuretar_models import ZUR_G


def _key(config, lens, dtype="bfloat16"):
    """The graph key of a step of fresh prompts of these lengths."""
    arch = resolve_architecture(config)
    rt = SimpleNamespace(dtype=dtype)
    ctx = SimpleNamespace(rt=rt, T=sum(lens), R=len(lens), n_want=len(lens), max_q_len=max(lens), max_keys=max(lens),
                          n_decode=sum(n == 1 for n in lens), decode_ordered=False)
    return Engine._graph_key(SimpleNamespace(model=Model(arch.build_plan(arch.config_class.from_dict(config)), rt)), ctx)[0]


# as many tokens and requests, longest portions in one run of 128 tokens; on either side of what the recurrence of the delta
# layer (first two) or of the linear attention (last) goes in chunks from
@pytest.mark.parametrize("walk,chunks", [((134, 133, 133), (240, 80, 80)), ((129, 129, 129, 113), (250, 90, 80, 80)), ((80, 76, 75), (127, 40, 64))])
def test_a_recurrence_in_chunks_has_a_graph_of_its_own(walk, chunks):
    assert _key(ZUR_G, walk) != _key(ZUR_G, chunks)
    assert _key(ZUR_G, walk, "float32") == _key(ZUR_G, chunks, "float32")          # (always token by token there)
    assert _key(ZUR_G, walk) == _key(ZUR_G, walk[::-1])


@pytest.mark.parametrize("few,many", [((55, 55), (100, 10)), ((5, 5), (8, 2)), ((16, 16), (17, 15)), ((130, 130), (145, 115))])
def test_tiles_of_queries_are_part_of_the_key(few, many):
    """Talking-heads attention sizes its grid (and a tile's buffers) by the longest portion: a graph captured for fewer
    tiles would leave the last queries of a longer portion undone."""
    assert _key(BUB_B, few) != _key(BUB_B, many)
    assert _key(BUB_B, few, "float32") == _key(BUB_B, many, "float32")             # (a block a token there)
    assert _key(BUB_B, (100, 100)) == _key(BUB_B, (104, 96))                       # (seven tiles each)
