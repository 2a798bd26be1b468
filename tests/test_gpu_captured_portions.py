"""Replayed step graphs whose spans are long enough for the kernels that run a span in chunks or in tiles.

A captured step launches what its bucket's rows and spans allow, with the choice between a layer's kernels made from the spans on
the device.  Here a portion of 300 to 420 rows (2100 for the scan) runs beside nine decoding requests, again and again: from the third
time on the bucket's graph is replayed with other lengths than it was captured with.  Logits against a runner without graphs."""
import random

import numpy as np
import pytest

import lolivik_configs as L
import traces
import vunolorn_configs as V
import zikevik_configs as Z
from zig_ai_b200.config import config_from_dict
from zig_ai_b200.weights import write_random_model

pytestmark = pytest.mark.gpu

MODELS = {
    "delta": (V.config(500, 128, 4.0, 1e-6, [V.delta(4, 2, 64, 128, 4, ff=256)]), 64),
    "delta_channel": (Z.config(500, 128, 1e-6, 1.0, [Z.delta(4, 2, 64, 128, 4, 16, 16, mlp=Z.dense(256))]), 64),
    "delta_small": (V.config(500, 128, 4.0, 1e-6, [V.delta(4, 2, 16, 32, 4, ff=256)]), 16),
    "latent": (Z.config(500, 256, 1e-6, 1.0, [Z.latent(16, 48, 32, 64, 256, 96, 0.1, 10000.0, mlp=Z.dense(256))]), 64),
    "memory": (L.config(500, 128, 1e-6, 0.7, [L.memory(4, 64, 64, 13.0, mlp=L.dense(256))]), 64),
    "shaped": (L.config(500, 256, 1e-6, 0.7, [L.attention(8, 2, 64, 64, 0.125, 25.0, 32, 1000, 0.25, 64, v_mix=False, mlp=L.dense(256))]), 64),
    "scan": (V.config(500, 128, 4.0, 1e-6, [V.mamba(256, 16, 8, 4, ff=256)]), 64),
}


@pytest.mark.parametrize("name", list(MODELS))
def test_portions_in_replayed_steps(name, tmp_path):
    from zig_ai_b200.engine.runner import load_runner
    cfg, page_size = MODELS[name]
    d = str(tmp_path / "m")
    write_random_model(config_from_dict(cfg), 11, d, matrix_std="fan_in")
    g = random.Random(5)
    rounds = [2100, 2060, 2095, 2081] if name == "scan" else [400, 421, 388, 390, 413]       # one bucket: rows in 64s
    runners = [load_runner(d, "bfloat16", max_tokens=16384, page_size=page_size, max_requests=16, graphs=graphs) for graphs in (True, False)]
    decoding = [(f"d{i}", [g.randrange(500) for _ in range(20 + 7 * i)]) for i in range(9)]
    portions = [[g.randrange(500) for _ in range(n)] for n in rounds]
    more = [[g.randrange(500) for _ in range(9)] for _ in rounds]
    outs = []
    for r in runners:
        got = []
        for k, toks in decoding:
            r.add_request(k)
            r.step([(k, toks, [len(toks) - 1])])
        for i, (toks, new) in enumerate(zip(portions, more)):
            r.add_request(f"p{i}")
            last = len(toks) - 1
            entries = [(k, [t], [0]) for (k, _), t in zip(decoding, new)] + [(f"p{i}", toks, sorted({0, 63, 64, 200, last}))]
            got.append(r.step(entries).float().cpu().numpy().copy())
            # the portion's state or pages, seen by its next tokens
            got.append(r.step([(f"p{i}", toks[:3], [0, 1, 2])]).float().cpu().numpy().copy())
            r.end_request(f"p{i}")
        outs.append(np.concatenate(got))
    assert runners[0].shape_graphs.replays >= len(rounds) - 3 + 1
    assert np.isfinite(outs[0]).all()
    # two ways of launching one step, whose products the library may sum in another order at the bucket's rounded row count; a span that
    # was lost, walked twice or read another's state moves a row by tens of per cent
    traces.check_same(outs[0], outs[1], "bfloat16", name, bf16_row=5e-2, bf16_mean=2e-2)
