"""Steps of single tokens through the recurrences' pass over the states (gla_step_kernel, delta_step_kernel) against the scans
that walk tokens, over state sizes around the pass's rows and columns, and with slots that were used before."""
import numpy as np
import pytest

import dabodra_util as db
import mulenex_util as mx
import nagilix_util as ng
import nomanex_util as nx
import soselix_util as sx
import zinavik_util as zv
from nomanex_util import open_engine, rel_err, write_model_dir

pytestmark = pytest.mark.gpu

FORMS = {
    "gla": (nx, lambda d, v: nx.make_config([(nx.gla(heads=3, dim=d, vdim=v), None)], width=64)),
    "mlstm": (mx, lambda d, v: mx.make_config([mx.layer(mx.mlstm(heads=3, dim=d, vdim=v), mlp=None)], width=64)),
    "hgrn2": (sx, lambda d, v: sx.make_config([sx.hgrn2(heads=3, dim=d, vdim=v, mlp=None)], width=64)),
    "mamba2": (sx, lambda d, v: sx.make_config([sx.mamba2(heads=4, vdim=v, state=d, groups=2, norm_groups=2, mlp=None)], width=64)),
    "constant decay": (zv, lambda d, v: zv.make_config([zv.layer(r=zv.right(heads=2, dim=d, vdim=v), mlp=None)], width=64)),
    "retention": (ng, lambda d, v: ng.make_config([ng.parallel(r=ng.right(heads=2, dim=d, vdim=v), mlp=None)], width=64)),
    "delta": (db, lambda d, v: db.make_config([db.delta(heads=4, kv_heads=2, dim=d, vdim=v, mlp=None)], width=64)),
}


@pytest.mark.parametrize("dim,vdim", [(4, 4), (16, 64), (17, 68), (64, 60), (65, 128), (128, 132), (130, 8), (256, 64), (258, 64), (64, 62)])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_single_tokens_equal_the_scan(tmp_path, monkeypatch, form, dim, vdim):
    util, make = FORMS[form]
    if form == "retention" and dim % 2:
        dim += 1
    cfg = make(dim, vdim)
    W = util.random_weights(cfg, seed=dim + vdim)
    d = write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(dim).integers(0, cfg["vocab"], (3, 40))
    out = {}
    for knob in ("1", "0"):
        monkeypatch.setenv("B200_SCAN_STEP", knob)
        with open_engine(d, dtype="bfloat16", max_seqs=3) as e:
            got = []
            for begin in (1, 4):               # the second round starts on the states that the first one left
                ids = [e.feed_open() for _ in range(3)]
                got.append(e.feed_step([(r, x[:begin], [begin - 1]) for r, x in zip(ids, t)]))
                for s in range(begin, begin + 9):
                    got.append(e.feed_step([(r, x[s:s + 1], [0]) for r, x in zip(ids, t)]))
                for r in ids:
                    e.feed_close(r)
            out[knob] = np.concatenate(got)
    # the states are the same bits; an output's sum over the state's rows, in fp32 and in another order, moves a rounding to
    # bf16 now and then
    r = rel_err(out["1"], out["0"].astype(np.float64))
    assert np.median(r) < 2.0 ** -9 and r.max() < 2.0 ** -5, (np.median(r), r.max())
