"""What captured step graphs are told apart by (no GPU): steps that share a key take the same launches."""
from types import SimpleNamespace

import pytest

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
