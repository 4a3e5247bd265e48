"""Attention of single tokens over bf16 rows of whole pieces (window_attn_rows_kernel) and the head preparation in front of it
(qk_prep_vec_kernel): against the general kernels and the oracles, over group sizes, head widths, windows, kept tokens,
sinks, caps and both kinds of gate, with contexts around a round of keys (64); and the same bits however many heads share a CTA."""
import numpy as np
import pytest

import dabodra_util as db
import mulenex_util as mx
import zinavik_util as zv
from nomanex_util import feed_portions, open_engine, rel_err, write_model_dir

pytestmark = pytest.mark.gpu
PORTIONS = [1, 1, 13, 1, 30, 1, 1, 15, 1, 1] + [31, 30, 1, 1, 1, 1, 2] + [7, 1, 1]   # 0 .. 141: no portion takes the 64-row kernel


def mulenex(heads, kv_heads, dim, vdim, tweak):
    return mx, mx.make_config([mx.layer(mx.attention(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, softcap=4.0 if tweak else None), mlp=None),
                               mx.layer(mx.attention(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim), mlp=None)], width=64)


def zinavik(heads, kv_heads, dim, vdim, tweak):
    return zv, zv.make_config([zv.layer(l=zv.left(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, window=33 if tweak else 500, keep_first=5 if tweak else 0,
                                                 rot_dims=dim // 2 if tweak else dim), mlp=None)], width=64)


def dabodra(heads, kv_heads, dim, vdim, tweak):
    return db, db.make_config([db.attention(heads=heads, kv_heads=kv_heads, dim=dim, window=17 if tweak else 300, rot_dims=dim // 2, mlp=None)], width=64)


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(16, 4, 128, 128), (8, 1, 64, 64), (2, 2, 8, 8), (6, 2, 40, 24), (6, 3, 32, 128), (12, 1, 120, 16)])
@pytest.mark.parametrize("make", [mulenex, zinavik, dabodra])
@pytest.mark.parametrize("tweak", [False, True])
def test_rows_of_keys_equal_the_general_kernel(tmp_path, monkeypatch, make, heads, kv_heads, dim, vdim, tweak):
    util, cfg = make(heads, kv_heads, dim, vdim, tweak)
    W = util.random_weights(cfg, seed=heads + dim)
    d = write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(dim).integers(0, cfg["vocab"], sum(PORTIONS)).tolist()
    out = {}
    for knob in ("1", "0"):
        monkeypatch.setenv("B200_WATTN_ROWS", knob)     # wherever they take the sizes, and nowhere
        monkeypatch.setenv("B200_QK_ROWS", knob)
        with open_engine(d, dtype="bfloat16") as e:
            out[knob] = feed_portions(e, t, PORTIONS)
    want = util.oracle_for(cfg, W).forward(t)
    a, b = (rel_err(out[k], want) for k in ("1", "0"))
    # bf16 projections, heads and residuals: up to ten roundings of 2^-9 of a value's size on the way to a row's logits, and scores of
    # rounded keys behind an exponential
    assert np.median(a) < 0.02 and a.max() < 0.06, (np.median(a), a.max())
    # both keep scores, weights and sums in fp32 and round once: neither may be further from the oracle than the other's roundings
    assert np.median(a) < 1.1 * np.median(b) + 2.0 ** -11 and a.max() < 2 * b.max() + 2.0 ** -8, (np.median(a), np.median(b), a.max(), b.max())
    assert np.median(rel_err(out["1"], out["0"].astype(np.float64))) < 0.012


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,together", [(16, 4, 128, 128, 2), (32, 8, 64, 64, 4), (64, 8, 32, 32, 8), (12, 1, 120, 16, 1)])
@pytest.mark.parametrize("tweak", [False, True])
def test_a_row_does_not_depend_on_how_many_heads_share_its_cta(tmp_path, monkeypatch, heads, kv_heads, dim, vdim, together, tweak):
    """48 sequences put `together` heads of a group to a CTA, one sequence one.  Everything else of a row is the same in both: products of up
    to 48 rows sum in an order that depends on the matrix alone, norms and preparation go row by row.  So the logits are the same bits."""
    assert (48 * heads // together >= 2 * 148 or together == 1) and (48 * heads // (2 * together) < 2 * 148 or heads // kv_heads % (2 * together) or together == 8)
    monkeypatch.setenv("B200_WATTN_ROWS", "1")
    util, cfg = mulenex(heads, kv_heads, dim, vdim, tweak)
    W = util.random_weights(cfg, seed=heads + dim)
    d = write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(dim).integers(0, cfg["vocab"], (48, 75)).tolist()
    with open_engine(d, dtype="bfloat16", max_seqs=48, max_tokens=128) as e:
        ids = [e.feed_open() for _ in t]
        many = [e.feed_step([(r, x[:1], [0]) for r, x in zip(ids, t)])] + [e.feed_step([(r, x[n:n + 1], [0]) for r, x in zip(ids, t)]) for n in range(1, 75)]
        for r in ids:
            e.feed_close(r)
        for i in (0, 47):
            alone = feed_portions(e, t[i], [1])
            assert np.array_equal(np.stack([m[i] for m in many]), alone), i
