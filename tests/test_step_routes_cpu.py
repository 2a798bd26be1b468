"""The host's rules for which kernels a step's spans take, and for the scratch that goes with them."""
import random
from types import SimpleNamespace

import pytest

from zig_ai_b200.kernels import ops


def step_of(q_lens, captured=False):
    return SimpleNamespace(q_lens=q_lens, n_seqs=len(q_lens), n_tokens=sum(q_lens), attn_tiles=sum(q_lens) // 128 + len(q_lens) if captured else None,
                           decode_only=all(n == 1 for n in q_lens))


def test_chunk_scratch_holds_every_chunk_and_little_more():
    g = random.Random(1)
    for _ in range(3000):
        cut, rows = g.choice([1, 24, 64, 128, 256, 1024]), g.choice([16, 64])
        q_lens = [g.choice([0, 1, 1, 1, g.randint(0, 300), cut, cut - 1, cut + 1, 64, 65]) for _ in range(g.randint(1, 40))]
        chunks = sum(-(-n // rows) for n in q_lens if n >= cut)
        assert ops._chunk_bound(step_of(q_lens), cut, rows) == chunks
        assert ops._chunk_bound(step_of(q_lens, True), cut, rows) >= chunks
    # one portion beside decoding requests, as a captured shape sees it (its spans rounded up): no chunk a request
    assert ops._chunk_bound(step_of([1] * 64 + [2048] + [0] * 63, True), 128, 64) == 33 + 16
    assert ops._chunk_bound(step_of([1] * 256 + [2048]), 128, 64) == 32


@pytest.mark.parametrize("cut", [lambda h, d, v: ops._delta_cut(h, d, v), lambda h, d, v: ops._mlstm_cut(d, v)])
def test_spans_take_their_kernels_by_the_layers_sizes_alone(cut):
    for h in (1, 4, 16, 64):
        for d in (1, 8, 16, 32, 64):
            for v in (1, 8, 33, 64, 128, 256):
                assert 64 <= cut(h, d, v) <= max(256, 32 * h)
