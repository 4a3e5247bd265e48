"""Attention of whole prompts (csrc/prompt_attention.cu) against the same tokens in portions (the kernels over the paged cache:
latent-space, window) and the oracles: lengths at the edges of its query and key tiles, windows from one key, one and more heads, sinks and
gates, several sequences in one step, and a sequence whose neighbour holds no finite number."""
import numpy as np
import pytest

import dabodra_util as db
import mulenex_util as mx
import nomanex_util as nx
import soselix_util as sx

pytestmark = pytest.mark.gpu

LENS = [32, 63, 64, 65, 127, 128, 129, 255, 256, 257, 320, 511, 513, 700]


def check(cfg, e, oracle, lens):
    rng = np.random.default_rng(len(lens))
    for n in lens:
        t = rng.integers(0, cfg["vocab"], n).tolist()
        new, old = nx.feed_whole(e, t), nx.feed_portions(e, t, [1, 20, 300])
        assert np.isfinite(new).all()
        # each form rounds queries or keys, weights, sums or values and the output to bf16 (2^-9 of a value at most, each): four
        # roundings a side, eight between the two
        r = nx.rel_err(new, old.astype(np.float64))
        assert np.median(r) < 8 * 2.0 ** -9 and r.max() < 10 * 8 * 2.0 ** -9, (n, np.median(r), r.max())
        want = oracle.forward(t)
        a, b = nx.rel_err(new, want), nx.rel_err(old, want)
        assert np.median(a) < 1.1 * np.median(b) + 2.0 ** -11, (n, np.median(a), np.median(b))


@pytest.mark.parametrize("heads,kv_rank", [(1, 128), (3, 136), (2, 512)])
def test_sinks_gates_and_shared_rows(tmp_path, heads, kv_rank):
    wide = dict(dim=128, rot_dim=64, vdim=128, kv_rank=kv_rank, q_rank=24, base=1000.0, mlp=None)
    cfg = sx.make_config([sx.latent(heads=heads, **wide), sx.latent(heads=heads + 1, kv_from=0, **wide)], width=32)
    W = sx.random_weights(cfg, seed=heads)
    with sx.open_engine(sx.write_model_dir(tmp_path / "m", cfg, W), dtype="bfloat16", max_tokens=1024) as e:
        check(cfg, e, sx.oracle_for(cfg, W), LENS if heads == 3 else LENS[:4])


@pytest.mark.parametrize("window", [1, 2, 64, 100, 129, 4096])
def test_windows(tmp_path, window):
    cfg = nx.make_config([(nx.latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=128, window=window, base=1000.0, rot_dims=32), None)], width=32)
    W = nx.random_weights(cfg, seed=window)
    with nx.open_engine(nx.write_model_dir(tmp_path / "m", cfg, W), dtype="bfloat16", max_tokens=1024) as e:
        check(cfg, e, nx.oracle_for(cfg, W), [65, 257, 700])


@pytest.mark.parametrize("heads,kv_heads,softcap,scale", [(1, 1, None, 0.09), (4, 2, 6.0, 0.2), (6, 2, 30.0, 1.0), (3, 3, None, 0.09)])
def test_caps_and_grouped_heads(tmp_path, heads, kv_heads, softcap, scale):
    wide = dict(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, scale=scale, softcap=softcap)
    cfg = mx.make_config([mx.layer(mx.attention(v_mix=False, **wide), mlp=None), mx.layer(mx.attention(**wide), mlp=None)], width=32)
    W = mx.random_weights(cfg, seed=heads)
    with mx.open_engine(mx.write_model_dir(tmp_path / "m", cfg, W), dtype="bfloat16", max_tokens=1024) as e:
        check(cfg, e, mx.oracle_for(cfg, W), LENS if heads == 4 else LENS[:4])


@pytest.mark.parametrize("window", [1, 65, 128, 4096])
def test_windows_and_sinks_over_grouped_heads(tmp_path, window):
    cfg = db.make_config([db.attention(heads=4, kv_heads=1, dim=128, window=window, rot_dims=32, base=1000.0, mlp=None)], width=32)
    W = db.random_weights(cfg, seed=window)
    with db.open_engine(db.write_model_dir(tmp_path / "m", cfg, W), dtype="bfloat16", max_tokens=1024) as e:
        check(cfg, e, db.oracle_for(cfg, W), [32, 65, 257, 700])


@pytest.mark.parametrize("design", ["soselix", "nomanex"])
def test_short_prompts_beside_a_long_one_are_no_less_exact(tmp_path, design):
    """The form is chosen by the mean length, so a step can hold prompts of a few tokens; and every prompt has first positions.
    Against the oracle they are as close as in the form that never rounds a value of its own."""
    wide = dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=128, base=1000.0)
    if design == "soselix":
        cfg = sx.make_config([sx.latent(q_rank=24, mlp=None, **wide)], width=64)
        W, oracle_for = sx.random_weights(cfg, seed=3), sx.oracle_for
    else:
        cfg = nx.make_config([(nx.latent(window=4096, **wide), None)], width=64)
        W, oracle_for = nx.random_weights(cfg, seed=3), nx.oracle_for
    oracle, new, old = oracle_for(cfg, W), [], []
    lens = [2, 3, 4, 6, 8, 12, 16, 24] * 4 + [1400]
    assert sum(lens) >= 32 * len(lens)
    with sx.open_engine(sx.write_model_dir(tmp_path / "m", cfg, W), dtype="bfloat16", max_tokens=1500, max_seqs=64, budget=4096, blocks=1024) as e:
        for seed in range(3):
            rng = np.random.default_rng(seed)
            seqs = [rng.integers(0, cfg["vocab"], n).tolist() for n in lens]
            want = np.concatenate([oracle.forward(s[:24]) for s in seqs])
            ids = [e.feed_open() for _ in seqs]
            new.append(e.feed_step([(r, s, list(range(min(24, len(s))))) for r, s in zip(ids, seqs)]) - want)
            old.append(np.concatenate([nx.feed_portions(e, s[:24], [1]) for s in seqs]) - want)
            for r in ids:
                e.feed_close(r)
    a, b = (np.sqrt((np.concatenate(v) ** 2).mean()) for v in (new, old))
    # 3 * 324 rows of 40 logits: the two root mean squares are each known to about 1 %
    assert a < 1.02 * b, (a, b)


def test_unequal_sequences_beside_one_without_finite_numbers(tmp_path):
    cfg = sx.make_config([sx.latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=128, q_rank=24, base=1000.0, mlp=None)], width=32)
    W = sx.random_weights(cfg, seed=9)
    d = sx.write_model_dir(tmp_path / "m", cfg, W)
    rng = np.random.default_rng(5)
    lens = [1, 300, 65, 40, 63, 2] + [int(n) for n in rng.integers(1, 180, 34)] + [257]
    assert sum(lens) >= 32 * len(lens)
    seqs = [rng.integers(1, cfg["vocab"], n).tolist() for n in lens]
    with sx.open_engine(d, dtype="bfloat16", max_tokens=400, max_seqs=64, budget=8192, blocks=2048) as e:
        alone = [nx.feed_portions(e, s, [1, 400])[-1] for s in seqs]
        ids = [e.feed_open() for _ in seqs]
        together = e.feed_step([(r, s, [len(s) - 1]) for r, s in zip(ids, seqs)])
        for r in ids:
            e.feed_close(r)
        r = nx.rel_err(together, np.stack(alone).astype(np.float64))
        assert np.median(r) < 8 * 2.0 ** -9 and r.max() < 80 * 2.0 ** -9, (np.median(r), r.max())
    W["embed"] = W["embed"].copy()
    W["embed"][0] = np.inf
    with sx.open_engine(sx.write_model_dir(tmp_path / "inf", cfg, W), dtype="bfloat16", max_tokens=400, max_seqs=64, budget=8192, blocks=2048) as e:
        seqs = [[0] * n if i % 3 == 2 else s for i, (s, n) in enumerate(zip(seqs, lens))]
        ids = [e.feed_open() for _ in seqs]
        got = e.feed_step([(r, s, [len(s) - 1]) for r, s in zip(ids, seqs)])
        for i in range(len(seqs)):
            if i % 3 != 2:
                np.testing.assert_array_equal(got[i], together[i])


@pytest.mark.parametrize("family", ["latent", "cap", "window"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_tokens_in_front_of_one_without_finite_numbers(tmp_path, family, bad):
    """A token whose values are not finite: what came before it, and what its window no longer reaches, does not depend on it."""
    if family == "latent":
        cfg = sx.make_config([sx.latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=128, q_rank=24, base=1000.0, mlp=None)], width=32)
        W = sx.random_weights(cfg, seed=9)
    elif family == "cap":
        cfg = mx.make_config([mx.layer(mx.attention(heads=4, kv_heads=2, dim=128, vdim=128, scale=0.2, softcap=6.0, v_mix=False), mlp=None)], width=32)
        W = mx.random_weights(cfg, seed=9)
    else:
        cfg = db.make_config([db.attention(heads=4, kv_heads=1, dim=128, window=65, rot_dims=32, base=1000.0, mlp=None)], width=32)
        W = db.random_weights(cfg, seed=9)
    W["embed"] = W["embed"].copy()
    for at in (1, 63, 64, 127, 128, 200, 255, 256, 300, 389):
        t = np.random.default_rng(at).integers(1, cfg["vocab"], 390)
        t[at] = 0
        out = []
        for row in (W["embed"][1].copy(), np.full(32, bad, dtype=np.float32)):
            W["embed"][0] = row
            with sx.open_engine(sx.write_model_dir(tmp_path / ("%d_%d" % (at, len(out))), cfg, W), dtype="bfloat16") as e:
                out.append(nx.feed_whole(e, t.tolist()))
        good = np.arange(390) < at
        if family == "window":
            good |= np.arange(390) >= at + 65
        assert np.isfinite(out[0]).all() and not np.isfinite(out[1][~good]).any(axis=-1).any()
        assert np.isfinite(out[1][good]).all(), (at, np.flatnonzero(good & ~np.isfinite(out[1]).all(axis=-1)))
        # rows formed again key by key: the same values without the roundings of weights and of the output's terms
        r = nx.rel_err(out[1][good], out[0][good].astype(np.float64))
        assert np.median(r) < 4 * 2.0 ** -9 and r.max() < 10 * 4 * 2.0 ** -9, (at, np.median(r), r.max())
