"""Norms between sublayers, embeddings and latent rows at widths around the edges of their pieces (csrc/hyper.cu, norm_act.cu,
latent_attention.cu): one, two and four pieces of four columns a thread, more than that, and rows that allow no wide access."""
import numpy as np
import pytest

import dabodra_util as dx
import mulenex_util as mx
import nomanex_util as nx
import soselix_util as sx

pytestmark = pytest.mark.gpu

WIDTHS = [4, 36, 252, 256, 260, 510, 516, 1020, 1028, 2044, 2052, 4096, 4100]


def model(family, width):
    if family == "mulenex":
        cfg = mx.make_config([mx.layer(mx.mlstm(heads=2, dim=16, vdim=8), mlp=None), mx.layer(mx.mlstm(heads=2, dim=16, vdim=8), mlp=None)], width=width)
        return cfg, mx.random_weights(cfg, seed=1), mx.oracle_for
    if family == "soselix":
        cfg = sx.make_config([sx.latent(q_rank=24, kv_rank=20, mlp=None), sx.hgrn2(mlp=None)], width=width)
        return cfg, sx.random_weights(cfg, seed=2), sx.oracle_for
    if family == "dabodra":
        cfg = dx.make_config([dx.attention(mlp=None), dx.delta(mlp=None)], width=width)
        return cfg, dx.random_weights(cfg, seed=3), dx.oracle_for
    cfg = nx.make_config([(nx.gla(), None), (nx.latent(), None)], width=width)
    return cfg, nx.random_weights(cfg, seed=4), nx.oracle_for


@pytest.mark.parametrize("family", ["mulenex", "soselix", "dabodra", "nomanex"])
@pytest.mark.parametrize("width", WIDTHS)
def test_rows_of_every_number_of_pieces(tmp_path, family, width):
    cfg, W, oracle = model(family, width)
    d = nx.write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(width).integers(0, cfg["vocab"], 21).tolist()
    want = oracle(cfg, W).forward(t)
    # fp32: sums of at most 4100 products, some sixty roundings of 2^-24 each where their signs are random, in about eight sublayers'
    # worth of operators: 3e-5; small widths divide by sums of few terms.  Nothing here routes, so that holds for every row
    with nx.open_engine(d) as e:
        assert nx.rel_err(nx.feed_whole(e, t), want).max() < 1e-4
        assert nx.rel_err(nx.feed_portions(e, t, [9] + [1] * 12), want).max() < 1e-4
    # bf16: eight operators' outputs rounded to 2^-9 of their size each.  A matrix memory's answer is a quotient, and where its divisor comes
    # near zero that moves the row and those behind it by more (width 516: four rows by 0.27 to 0.6)
    with nx.open_engine(d, dtype="bfloat16") as e:
        r = np.sort(nx.rel_err(nx.feed_portions(e, t, [9] + [1] * 12), want))
        assert np.median(r) < 0.06 and (r[15] < 0.1 if family == "mulenex" else r[-1] < 0.25), r[-6:]


@pytest.mark.parametrize("q_rank,kv_rank", [(1, 1), (127, 129), (1024, 512), (1025, 1023), (40, 1100)])
def test_latent_rows_that_stay_in_registers_and_longer_ones(tmp_path, q_rank, kv_rank):
    cfg = sx.make_config([sx.latent(heads=2, q_rank=q_rank, kv_rank=kv_rank, mlp=None)], width=32)
    W = sx.random_weights(cfg, seed=q_rank)
    d = nx.write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(5).integers(0, cfg["vocab"], 17).tolist()
    with nx.open_engine(d) as e:
        assert nx.rel_err(nx.feed_portions(e, t, [8] + [1] * 9), sx.oracle_for(cfg, W).forward(t)).max() < 1e-4


@pytest.mark.parametrize("ranks", [(24, 20), (130, 40)])
def test_latent_rows_of_more_tokens_than_stay_in_registers(tmp_path, ranks):
    """Both sides of the line for short rows (512 tokens): in a step of 600 rows are read again, in two of 300 they are held; the same sums."""
    cfg = sx.make_config([sx.latent(heads=2, q_rank=ranks[0], kv_rank=ranks[1], mlp=None)], width=32)
    W = sx.random_weights(cfg, seed=7)
    d = nx.write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(6).integers(0, cfg["vocab"], 600).tolist()
    with nx.open_engine(d, max_tokens=640) as e:
        whole, parts = nx.feed_whole(e, t), nx.feed_portions(e, t, [300])
    assert nx.rel_err(whole, sx.oracle_for(cfg, W).forward(t)).max() < 1e-4
    assert nx.rel_err(parts, whole.astype(np.float64)).max() < 1e-5


@pytest.mark.parametrize("taps", [2, 3, 4])
def test_short_convolution_over_sequences_that_end_inside_its_rounds(tmp_path, taps):
    """Rows come in rounds of four and walks of up to sixteen; sequences begin and end anywhere in them and go on from what they carry."""
    cfg = dx.make_config([dx.delta(heads=4, kv_heads=2, dim=8, vdim=8, conv=taps, mlp=None)], width=32)
    W = dx.random_weights(cfg, seed=taps)
    d = nx.write_model_dir(tmp_path / "m", cfg, W)
    rng = np.random.default_rng(taps)
    first = [1, 2, 3, 4, 5, 7, 16, 17, 1, 31, 6, 1, 1, 64, 3, 33]
    seqs = [rng.integers(0, cfg["vocab"], n + 1 + i % 5) for i, n in enumerate(first)]
    want = [dx.oracle_for(cfg, W).forward(s.tolist()) for s in seqs]
    for dtype, tol in (("float32", 1e-4), ("bfloat16", 0.06)):     # fp32 sums; three operators' outputs rounded to 2^-9 each
        with nx.open_engine(d, dtype=dtype, max_tokens=128, max_seqs=16, budget=512, blocks=128) as e:
            ids = [e.feed_open() for _ in seqs]
            a = e.feed_step([(r, s[:n].tolist(), [n - 1]) for r, s, n in zip(ids, seqs, first)])
            b = e.feed_step([(r, s[n:].tolist(), [len(s) - n - 1]) for r, s, n in zip(ids, seqs, first)])
        # every sequence: a fault at one kind of boundary touches few of the sixteen
        assert nx.rel_err(np.asarray(a), np.stack([w[n - 1] for w, n in zip(want, first)])).max() < tol
        assert nx.rel_err(np.asarray(b), np.stack([w[-1] for w in want])).max() < tol
