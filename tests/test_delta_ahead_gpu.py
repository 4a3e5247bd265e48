"""Delta-rule chunks on both sides of rules::delta_scores_ahead (csrc/delta_chunk.cu): sequences fed together, whose CTAs share the SMs and form their own
scores, against each of them alone, whose scores come a chunk ahead, and a whole sequence against its portions; one to six chunks, ends inside a block,
more sequences than are put in order.  And the two forms on the same step, bit by bit."""
import ctypes as C

import numpy as np
import pytest
import torch

import dabodra_util as db
import nomanex_util as nx

pytestmark = pytest.mark.gpu

SHAPES = [(8, 4, 16, 16), (8, 8, 128, 64), (8, 2, 112, 72), (8, 1, 48, 24), (8, 8, 64, 136)]
LENS = [65, 128, 129, 333, 64, 1, 200]


def model(tmp_path, heads, kv_heads, dim, vdim):
    cfg = db.make_config([db.delta(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, conv=4, mlp=None)], width=64, vocab=60)
    return db.write_model_dir(tmp_path / "m", cfg, db.random_weights(cfg, seed=dim, a_log=(-5.0, 0.0)))


def ahead(e, heads, vdim, lens):
    return e._l.b200_rule_query(12, (C.c_int32 * 5)(heads * -(-vdim // 64), len(lens), sum(lens), max(lens), torch.cuda.get_device_properties(0).multi_processor_count), 5)


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", SHAPES)
def test_sequences_together_equal_each_alone(tmp_path, monkeypatch, heads, kv_heads, dim, vdim):
    monkeypatch.setenv("B200_DELTA_CHUNK", "1")
    rng = np.random.default_rng(dim)
    lens = LENS * 11
    seqs = [rng.integers(0, 60, n).tolist() for n in lens]
    with db.open_engine(model(tmp_path, heads, kv_heads, dim, vdim), dtype="bfloat16", max_tokens=400, max_seqs=len(lens), budget=max(4096, sum(lens)), blocks=2048) as e:
        # the two sides this is about; a sequence of one chunk has nothing ahead
        assert not ahead(e, heads, vdim, lens) and all(ahead(e, heads, vdim, [n]) == (n > 64) for n in lens)
        ids = [e.feed_open() for _ in seqs]
        together = e.feed_step([(r, s, list(range(len(s)))) for r, s in zip(ids, seqs)])
        for r in ids:
            e.feed_close(r)
        alone = np.concatenate([nx.feed_whole(e, s) for s in seqs[:21]])
        parts = np.concatenate([nx.feed_portions(e, s, [130, 70, 66]) for s in seqs[:7]])
    # the recurrence keeps fp32 either way; products of other step sizes sum in other orders, and a rounding to bf16 moves now and then
    for a, b in ((together[:len(alone)], alone), (parts, alone[:len(parts)])):
        r = nx.rel_err(a, b.astype(np.float64))
        assert np.median(r) < 2.0 ** -9 and r.max() < 2.0 ** -5, (np.median(r), r.max())


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", SHAPES)
@pytest.mark.parametrize("lens", [[333], LENS, [64, 1, 63], LENS * 10])
def test_both_forms_give_the_same_bits(tmp_path, monkeypatch, heads, kv_heads, dim, vdim, lens):
    monkeypatch.setenv("B200_DELTA_CHUNK", "1")
    rng = np.random.default_rng(dim + len(lens))
    first, second = ([rng.integers(0, 60, n).tolist() for n in lens] for _ in range(2))
    out = []
    with db.open_engine(model(tmp_path, heads, kv_heads, dim, vdim), dtype="bfloat16", max_tokens=800, max_seqs=len(lens), budget=max(4096, sum(lens)), blocks=4096) as e:
        for form in "01":
            monkeypatch.setenv("B200_DELTA_AHEAD", form)
            ids = [e.feed_open() for _ in lens]
            # outputs of the first portions, and of second ones, which start from the states that the first left
            out.append([e.feed_step([(r, s, list(range(len(s)))) for r, s in zip(ids, seqs)]) for seqs in (first, second)])
            for r in ids:
                e.feed_close(r)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
