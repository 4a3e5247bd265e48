"""Delta-rule chunks on both sides of rules::delta_scores_ahead (csrc/delta_chunk.cu): sequences fed together, whose CTAs share the SMs and form their own
scores, against each of them alone, whose scores come a chunk ahead, and a whole sequence against its portions; one to six chunks, ends inside a block,
more sequences than are put in order."""
import numpy as np
import pytest

import dabodra_util as db
import nomanex_util as nx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(8, 4, 16, 16), (8, 8, 128, 64), (8, 2, 112, 72), (8, 1, 48, 24), (8, 8, 64, 136)])
def test_sequences_together_equal_each_alone(tmp_path, monkeypatch, heads, kv_heads, dim, vdim):
    monkeypatch.setenv("B200_DELTA_CHUNK", "1")
    cfg = db.make_config([db.delta(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, conv=4, mlp=None)], width=64, vocab=60)
    W = db.random_weights(cfg, seed=dim, a_log=(-5.0, 0.0))
    rng = np.random.default_rng(dim)
    lens = [65, 128, 129, 333, 64, 1, 200] * (3 if dim < 128 else 11)
    seqs = [rng.integers(0, 60, n).tolist() for n in lens]
    with db.open_engine(db.write_model_dir(tmp_path / "m", cfg, W), dtype="bfloat16", max_tokens=400, max_seqs=len(lens), budget=max(4096, sum(lens))) as e:
        ids = [e.feed_open() for _ in seqs]
        together = e.feed_step([(r, s, list(range(len(s)))) for r, s in zip(ids, seqs)])
        for r in ids:
            e.feed_close(r)
        alone = np.concatenate([nx.feed_whole(e, s) for s in seqs])
        parts = np.concatenate([nx.feed_portions(e, s, [130, 70, 66]) for s in seqs[:7]])
    # the recurrence keeps fp32 either way; products of other step sizes sum in other orders, and a rounding to bf16 moves now and then
    for a, b in ((together, alone), (parts, alone[:len(parts)])):
        r = nx.rel_err(a, b.astype(np.float64))
        assert np.median(r) < 2.0 ** -9 and r.max() < 2.0 ** -5, (np.median(r), r.max())
