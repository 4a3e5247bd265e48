"""Expert choice with scores in registers (csrc/moe.cu) at the sizes where another number of registers or the scratch row takes over, groups held by
one lane and by two, and steps whose pairs outgrow the sort's registers, against the oracle through a model of one layer."""
import numpy as np
import pytest

import mulenex_util as mx
import nomanex_util as nx

pytestmark = pytest.mark.gpu


def check(mod, d, cfg, W, tokens, top):
    t = np.random.default_rng(top).integers(0, cfg["vocab"], tokens).tolist()
    with mod.open_engine(d, max_tokens=512, budget=512) as e:
        r = nx.rel_err(nx.feed_whole(e, t), mod.oracle_for(cfg, W).forward(t))
    # fp32 sums of a few dozen products: 1e-6 of a row; a wrong expert changes tenths of it
    assert r.max() < 1e-3, r.max()


@pytest.mark.parametrize("experts,top", [(1, 1), (31, 3), (32, 32), (33, 5), (64, 2), (65, 7), (128, 4), (129, 6), (256, 30), (257, 3), (40, 33)])
@pytest.mark.parametrize("tokens", [3, 400])
def test_experts_around_a_register_and_the_scratch_row(tmp_path, experts, top, tokens):
    cfg = mx.make_config([mx.layer(mx.attention(heads=2, kv_heads=1, dim=8, vdim=6), mlp=mx.moe(experts=experts, top=top, ff=8))], width=32)
    W = mx.random_weights(cfg, seed=experts)
    check(mx, mx.write_model_dir(tmp_path / "m", cfg, W), cfg, W, tokens, top)


@pytest.mark.parametrize("experts,count,keep,top", [(32, 32, 3, 3), (66, 33, 2, 4), (128, 64, 40, 6), (256, 8, 3, 8), (48, 3, 1, 16), (24, 4, 4, 5)])
def test_groups_of_experts(tmp_path, experts, count, keep, top):
    cfg = nx.make_config([(nx.gla(), nx.moe(experts=experts, top=top, count=count, keep=keep))], width=32)
    W = nx.random_weights(cfg, seed=experts)
    check(nx, nx.write_model_dir(tmp_path / "m", cfg, W), cfg, W, 100, top)
