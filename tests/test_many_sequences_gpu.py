"""Steps of many sequences: the tables of (sequence, tile) looked up 32 sequences at a time, per-head products in blocks of 16 rows,
the combine of fp32 expert rows - every sequence against the oracle, whatever shares its step."""
import numpy as np
import pytest

import mulenex_util as mx
import soselix_util as sx
from nomanex_util import open_engine, rel_err, write_model_dir

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seqs", [17, 32, 33, 65, 100])
def test_latent_steps_of_many_sequences(tmp_path, seqs):
    cfg = sx.make_config([sx.latent(heads=4, dim=16, rot_dim=16, vdim=32, kv_rank=48, q_rank=24, mlp=None)], width=64)
    W = sx.random_weights(cfg, seed=seqs)
    d = write_model_dir(tmp_path / "m", cfg, W)
    oracle = sx.oracle_for(cfg, W)
    n = [1 + (7 * i) % 3 for i in range(seqs)]
    t = [np.random.default_rng(i).integers(0, cfg["vocab"], k + 3).tolist() for i, k in enumerate(n)]
    with open_engine(d, dtype="bfloat16", max_seqs=seqs) as e:
        ids = [e.feed_open() for _ in t]
        got = [e.feed_step([(r, x[:k], [k - 1]) for r, x, k in zip(ids, t, n)])]
        for s in range(3):
            got.append(e.feed_step([(r, x[k + s:k + s + 1], [0]) for r, x, k in zip(ids, t, n)]))
    for i, (x, k) in enumerate(zip(t, n)):
        want = np.asarray(oracle.forward(x))[k - 1:]
        r = rel_err(np.stack([g[i] for g in got]), want)
        # bf16 roundings of one layer and of the head on a width of 64: a few percent of a row
        assert r.max() < 0.1, (i, r)


@pytest.mark.parametrize("seqs", [31, 40, 67])
def test_window_portions_of_many_sequences(tmp_path, seqs):
    cfg = mx.make_config([mx.layer(mx.attention(heads=4, kv_heads=2, dim=16, vdim=16), mlp=mx.moe(experts=4, top=2, ff=16, shared=16))], width=64)
    W = mx.random_weights(cfg, seed=seqs)
    d = write_model_dir(tmp_path / "m", cfg, W)
    oracle = mx.oracle_for(cfg, W)
    n = [3 + (5 * i) % 17 for i in range(seqs)]
    t = [np.random.default_rng(i).integers(0, cfg["vocab"], 2 * k).tolist() for i, k in enumerate(n)]
    with open_engine(d, dtype="bfloat16", max_seqs=seqs, max_tokens=64, budget=1024) as e:
        ids = [e.feed_open() for _ in t]
        got = [e.feed_step([(r, x[a * k:(a + 1) * k], [k - 1]) for r, x, k in zip(ids, t, n)]) for a in (0, 1)]
    r = np.array([rel_err(np.stack([g[i] for g in got]), np.asarray(oracle.forward(x))[[k - 1, 2 * k - 1]]) for i, (x, k) in enumerate(zip(t, n))])
    # a routing choice that rounding turns moves its row; the others show the roundings of two layers
    assert np.median(r) < 0.05 and np.quantile(r, 0.9) < 0.2, (np.median(r), np.quantile(r, 0.9))
