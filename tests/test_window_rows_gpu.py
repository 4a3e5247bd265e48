"""Attention of single tokens over bf16 rows of whole pieces (window_attn_rows_kernel) and the head preparation in front of it
(qk_prep_vec_kernel): against the general kernels' results and the oracles, over group sizes, head widths, windows, kept tokens,
sinks, caps and both kinds of gate, with contexts around a round of keys (128), and the same whatever shares the batch."""
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
        monkeypatch.setenv("B200_WATTN_ROWS", knob)
        with open_engine(d, dtype="bfloat16", max_seqs=41) as e:
            out[knob] = feed_portions(e, t, PORTIONS)
            if knob == "1":
                # 40 sequences of one length side by side (more heads to a CTA), then the same tokens alone: equal to the bit
                ids = [e.feed_open() for _ in range(40)]
                many = [e.feed_step([(r, t[a:a + n], [n - 1]) for r in ids]) for a, n in ((0, 1), (1, 1), (2, 1))]
                for r in ids:
                    e.feed_close(r)
                one = e.feed_open()
                for step, (a, n) in zip(many, ((0, 1), (1, 1), (2, 1))):
                    alone = e.feed_step([(one, t[a:a + n], [n - 1])])
                    # projections of 40 rows and of one row sum in other orders: the same within their roundings
                    assert (rel_err(step, np.repeat(alone.astype(np.float64), 40, 0)) < 0.05).all()
                    assert (step == step[:1]).all()
                e.feed_close(one)
    want = util.oracle_for(cfg, W).forward(t)
    a, b = (rel_err(out[k], want) for k in ("1", "0"))
    # both keep scores, weights and sums in fp32 and round once: neither may be further from the oracle than the other's roundings
    assert np.median(a) < 1.1 * np.median(b) + 2.0 ** -11 and a.max() < 2 * b.max() + 2.0 ** -8, (np.median(a), np.median(b), a.max(), b.max())
    assert np.median(rel_err(out["1"], out["0"].astype(np.float64))) < 0.012
