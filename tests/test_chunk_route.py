"""Which steps a recurrence with one decay per head takes in chunks of tokens, and from how many tokens of a request on; and that
captured steps on the two sides of its lines are different graphs, for models that have such layers and for no others."""

from types import MethodType, SimpleNamespace

import pytest
import torch

from clockwork_b200.engine.step import ModelRunner, StepEntry
from clockwork_b200.parts.state_mixers import CHUNKS_BESIDE_FROM, CHUNKS_FROM, takes_chunks

BF16, F32 = SimpleNamespace(dtype=torch.bfloat16), SimpleNamespace(dtype=torch.float32)


def context(tokens, longest, lens, extras):
    return SimpleNamespace(num_tokens=tokens, max_q_len=longest, all_single_token=longest <= 1, q_lens_host=lens, extras=extras)


@pytest.mark.parametrize("lens, want, short", [
    ([1, 1, 1], 0, 0), ([CHUNKS_FROM - 1], 0, 0), ([40] * 6, 0, 0), ([CHUNKS_FROM - 1] + [1] * 200, 0, 0),  # no portion long enough
    ([64] * 4, 0, 1), ([32] * 8, 0, 1),  # .. in a long step: chunks for the layers that ask for it
    ([CHUNKS_FROM], 1, 1), ([900, 333, 65], 1, 1), ([2, CHUNKS_FROM], 1, 1),
    ([CHUNKS_FROM, 1], 0, 0), ([CHUNKS_BESIDE_FROM - 25] + [1] * 24, 0, 0),  # too few tokens for a launch beside the single tokens'
    ([CHUNKS_BESIDE_FROM - 24] + [1] * 24, 2, 2), ([391, 130] + [1] * 24, 2, 2),  # single tokens keep to the scan of steps of single tokens
])
def test_eager_steps(lens, want, short):
    ctx = context(sum(lens), max(lens), lens, {})
    assert takes_chunks(BF16, ctx) == want and takes_chunks(BF16, ctx, short_portions=True) == short
    assert takes_chunks(F32, ctx) == takes_chunks(F32, ctx, short_portions=True) == 0


@pytest.mark.parametrize("tokens, singles, portions, want, short", [(64, False, 0, 0, 0), (128, False, 2, 1, 1), (256, False, 1, 0, 1), (192, True, 2, 0, 0),
                                                                    (256, True, 2, 2, 2), (1024, True, 1, 0, 0), (1024, False, 2, 1, 1)])
def test_captured_steps(tokens, singles, portions, want, short):
    ctx = context(tokens, tokens, [], {"captured_portions": {"singles": singles, "long": portions}})
    assert takes_chunks(BF16, ctx) == want and takes_chunks(BF16, ctx, short_portions=True) == short and takes_chunks(F32, ctx) == 0


@pytest.mark.parametrize("long_from", [0, CHUNKS_FROM])
def test_keys_of_captured_steps(long_from):
    runner = SimpleNamespace(portions_captured=True, graph_max_ctx=4096, long_portions_from=long_from,
                             cache=SimpleNamespace(get=lambda _: SimpleNamespace(num_computed=0)), model=SimpleNamespace(spec=SimpleNamespace(vocab_size=1000)))
    for name in ("PORTION_SEQ_BUCKETS", "PORTION_TOKEN_BUCKETS", "PORTION_MAX_LOGITS", "PORTION_MAX_PORTIONS", "PORTION_LONG_STEP", "PORTION_MAX_TOKENS",
                 "PORTION_LONG_WASTE"):
        setattr(runner, name, getattr(ModelRunner, name))
    runner._portion_token_bucket = MethodType(ModelRunner._portion_token_bucket, runner)
    key = lambda *lens: ModelRunner._portion_graph_key(runner, [StepEntry(str(i), [1] * n, [n - 1]) for i, n in enumerate(lens)])  # noqa: E731
    assert key(120)[:5] == key(40, 40, 40)[:5] == (128, 8, 8, 1024, False)
    assert (key(120) != key(40, 40, 40)) == (key(70, 70, 70) != key(210)) == bool(long_from)
    assert key(120) == key(100, 20) and key(60) == key(30, 30)
    classes = [key(*lens)[5] for lens in ([CHUNKS_FROM - 1], [70, 70], [70, 70, 70], [CHUNKS_FROM], [700])]
    assert classes == ([0, 0, 1, 2, 2] if long_from else [0] * 5)
