"""The recurrent scan with its chunks side by side (csrc/scan_parallel.cu) against the token-by-token scan and the oracles: head
sizes at the edges of its tiles, portions that end inside blocks and chunks, states that come in and go out, decays from none
to complete."""
import numpy as np
import pytest

import mulenex_util as mx
import nomanex_util as nx
import soselix_util as sx

pytestmark = pytest.mark.gpu

PORTIONS = [100, 64, 1, 17, 2, 128, 15, 1]


def both(d, t, monkeypatch, max_tokens=400):
    out = {}
    for knob in ("1", "0"):          # from one token per portion; never
        monkeypatch.setenv("B200_SCAN_CHUNK", knob)
        with nx.open_engine(d, dtype="bfloat16", max_tokens=max_tokens) as e:
            out[knob] = (nx.feed_whole(e, t), nx.feed_portions(e, t, PORTIONS))
    return out["1"], out["0"]


def check(new, old, want):
    # both scans are fp32; behind them the layer's output is rounded to bf16 (2^-8 of a value at most), so the logits differ by the
    # few roundings that fall the other way
    for a, b in zip(new, old):
        assert np.isfinite(a).all()
        r = nx.rel_err(a, b.astype(np.float64))
        assert np.median(r) < 2e-3 and r.max() < 2e-2, (np.median(r), r.max())
        assert np.median(nx.rel_err(a, want)) < 1.05 * np.median(nx.rel_err(b, want)) + 2e-4


@pytest.mark.parametrize("heads,dim,vdim", [(1, 16, 8), (2, 48, 24), (3, 128, 128), (2, 64, 136), (1, 112, 200), (2, 128, 64)])
@pytest.mark.parametrize("bias", [9.0, 2.0, -4.0, -300.0])
def test_gated_linear_attention(tmp_path, monkeypatch, heads, dim, vdim, bias):
    cfg = nx.make_config([(nx.gla(heads=heads, dim=dim, vdim=vdim, tau=4.0), None)], width=32)
    W = nx.random_weights(cfg, seed=3)
    W["l0.mix.a2.b"] = nx.bf16_round(W["l0.mix.a2.b"] - 2.0 + bias)          # from nearly no decay to nothing left of the past
    d = nx.write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(1).integers(0, cfg["vocab"], 330).tolist()
    new, old = both(d, t, monkeypatch)
    check(new, old, nx.oracle_for(cfg, W).forward(t))


@pytest.mark.parametrize("heads,dim,vdim", [(2, 16, 8), (1, 80, 40), (2, 128, 128), (1, 96, 264)])
@pytest.mark.parametrize("bias,lower", [(1.0, (0.0, 0.9)), (-12.0, (0.0, 0.0)), (14.0, (0.0, 0.0)), (-40.0, (0.0, 0.999))])
def test_hgrn2(tmp_path, monkeypatch, heads, dim, vdim, bias, lower):
    cfg = sx.make_config([sx.hgrn2(heads=heads, dim=dim, vdim=vdim, mlp=None)], width=32)
    W = sx.random_weights(cfg, seed=4, lower=lower)
    W["l0.mix.f.b"] = sx.bf16_round(W["l0.mix.f.b"] - 1.0 + bias)
    d = sx.write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(2).integers(0, cfg["vocab"], 330).tolist()
    new, old = both(d, t, monkeypatch)
    check(new, old, sx.oracle_for(cfg, W).forward(t))


@pytest.mark.parametrize("heads,dim,vdim", [(2, 16, 8), (1, 80, 40), (2, 128, 128), (1, 64, 136)])
@pytest.mark.parametrize("gate_bias", [(0.0, 2.0), (-8.0, 12.0), (8.0, -30.0)])
def test_mlstm(tmp_path, monkeypatch, heads, dim, vdim, gate_bias):
    cfg = mx.make_config([mx.layer(mx.mlstm(heads=heads, dim=dim, vdim=vdim, gate_cap=40.0), mlp=None)], width=32)
    W = mx.random_weights(cfg, seed=5, gate_bias=gate_bias)
    d = mx.write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(3).integers(0, cfg["vocab"], 330).tolist()
    new, old = both(d, t, monkeypatch)
    check(new, old, mx.oracle_for(cfg, W).forward(t))


def test_unequal_sequences_in_one_step_and_their_states(tmp_path, monkeypatch):
    """More sequences than a warp has lanes, some without a whole block; the next step starts from the states they left."""
    cfg = nx.make_config([(nx.gla(heads=2, dim=32, vdim=40, tau=8.0), None)], width=32)
    W = nx.random_weights(cfg, seed=6)
    d = nx.write_model_dir(tmp_path / "m", cfg, W)
    rng = np.random.default_rng(7)
    lens = [int(n) for n in rng.integers(1, 140, 40)] + [64, 65, 63, 128]
    seqs = [rng.integers(0, cfg["vocab"], n + 30).tolist() for n in lens]
    out = {}
    for knob in ("1", "0"):
        monkeypatch.setenv("B200_SCAN_CHUNK", knob)
        with nx.open_engine(d, dtype="bfloat16", max_tokens=200, max_seqs=64, budget=4096, blocks=1024) as e:
            ids = [e.feed_open() for _ in seqs]
            a = e.feed_step([(r, s[:n], [n - 1]) for r, s, n in zip(ids, seqs, lens)])
            b = e.feed_step([(r, s[n:], list(range(30))) for r, s, n in zip(ids, seqs, lens)])
            out[knob] = np.concatenate([a, b])
    r = nx.rel_err(out["1"], out["0"].astype(np.float64))
    assert np.median(r) < 2e-3 and r.max() < 2e-2, (np.median(r), r.max())


@pytest.mark.parametrize("family", ["hgrn2", "mlstm"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [1, 15, 16, 40, 63, 64, 70])
def test_tokens_in_front_of_one_without_finite_numbers(tmp_path, family, bad, at):
    """A token whose values are not finite, in every place of a block and a chunk: what came before it does not depend on it."""
    if family == "hgrn2":
        cfg = sx.make_config([sx.hgrn2(heads=2, dim=48, vdim=72, mlp=None)], width=32)
        W = sx.random_weights(cfg, seed=4)
    else:
        cfg = mx.make_config([mx.layer(mx.mlstm(heads=2, dim=48, vdim=72), mlp=None)], width=32)
        W = mx.random_weights(cfg, seed=4)
    W["embed"] = W["embed"].copy()
    t = np.random.default_rng(at).integers(1, cfg["vocab"], 90)
    t[at] = 0
    out = []
    for row in (W["embed"][1].copy(), np.full(32, bad, dtype=np.float32)):
        W["embed"][0] = row
        with sx.open_engine(sx.write_model_dir(tmp_path / ("m%d" % len(out)), cfg, W), dtype="bfloat16") as e:
            out.append(nx.feed_whole(e, t.tolist()))
    assert np.isfinite(out[0]).all() and not np.isfinite(out[1][at:]).all()
    np.testing.assert_array_equal(out[1][:at], out[0][:at])
