"""Mamba-2 prompts cut into segments that run side by side (csrc/scan_chunk.cu) against one chain of chunks a sequence: lengths around
the segment (256) and the chunk (64), state sizes around the fragments, portions that go on from a state."""
import numpy as np
import pytest

import soselix_util as sx
from nomanex_util import open_engine, rel_err, write_model_dir

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,groups,state,vdim", [(4, 2, 128, 64), (2, 1, 16, 72), (3, 3, 48, 8), (2, 2, 64, 136)])
@pytest.mark.parametrize("lens", [[1], [255], [256], [257], [512, 64], [65, 700, 256], [513, 1, 130, 300]])
def test_segments_equal_the_chain(tmp_path, monkeypatch, heads, groups, state, vdim, lens):
    cfg = sx.make_config([sx.mamba2(heads=heads, vdim=vdim, state=state, groups=groups, norm_groups=1, mlp=None)], width=64)
    W = sx.random_weights(cfg, seed=state)
    d = write_model_dir(tmp_path / "m", cfg, W)
    t = [np.random.default_rng(i).integers(0, cfg["vocab"], 2 * n + 1).tolist() for i, n in enumerate(lens)]
    out = {}
    for knob in ("1", "0"):
        monkeypatch.setenv("B200_SCAN_SEGMENTS", knob)
        monkeypatch.setenv("B200_SCAN_CHUNK", "1")
        with open_engine(d, dtype="bfloat16", max_seqs=4, max_tokens=2048, budget=2048) as e:
            ids = [e.feed_open() for _ in lens]
            got = [e.feed_step([(r, x[:n], list(range(n))) for r, x, n in zip(ids, t, lens)])]
            got.append(e.feed_step([(r, x[n:2 * n], list(range(n))) for r, x, n in zip(ids, t, lens)]))     # behind a state
            got.append(e.feed_step([(r, x[2 * n:], [0]) for r, x, n in zip(ids, t, lens)]))                 # and on the state left
            out[knob] = np.concatenate(got)
    # fp32 sums cut in other places: a rounding to bf16 moves now and then
    r = rel_err(out["1"], out["0"].astype(np.float64))
    assert np.median(r) < 2.0 ** -9 and r.max() < 2.0 ** -5, (np.median(r), r.max())
