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


def test_latent_attention_goes_where_the_keys_are():
    def cut(ctx, q_lens, heads=16, rank=256, captured=False):
        s = step_of(q_lens, captured)
        s.kv_lens = [c + n for c, n in zip(ctx, q_lens)]
        return ops._latent_cut(s, heads, rank, 32)
    # a span alone: by its rows, whatever its context
    for ctx in (0, 1000, 16000):
        assert cut([ctx], [64]) > 64 and cut([ctx], [128]) <= 128
    assert cut([4000], [32], heads=128) <= 32 and cut([4000], [128], rank=128) > 128
    # a few decoding requests far behind, beside a prompt's portion: their tiles would walk their keys alone
    assert cut([16000] * 12 + [0], [1] * 12 + [100]) > 100
    assert 1 < cut([16000] * 12 + [6000], [1] * 12 + [400]) <= 400
    assert cut([16000, 0], [20, 200]) > 20
    # many short spans together
    assert cut([500] * 16, [20] * 16) == 1
    # so many rows that mma.sync would not cut keys into ranges
    assert cut([16000] * 12 + [0], [1] * 12 + [1900]) == 1
    # contexts not known: each span by itself
    assert 100 < cut([16000] * 12 + [0], [1] * 12 + [200], captured=True) <= 200
