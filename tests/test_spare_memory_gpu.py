"""Workspaces of forms that a step can also do without are no reason to refuse an engine: where memory is short they stay away."""
import numpy as np
import pytest
import torch

import mulenex_util as mx
import nomanex_util as nx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("design", ["nomanex", "mulenex"])
def test_an_engine_without_room_for_them_is_created_and_right(tmp_path, design):
    if design == "nomanex":
        cfg = nx.make_config([(nx.gla(heads=16, dim=128, vdim=128), None), (nx.latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=128, window=64), None)], width=32)
        W, oracle = nx.random_weights(cfg, seed=1), nx.oracle_for
    else:
        cfg = mx.make_config([mx.layer(mx.mlstm(heads=16, dim=128, vdim=128), mlp=None), mx.layer(mx.attention(heads=4, kv_heads=2, dim=128, vdim=128), mlp=None)], width=32)
        W, oracle = mx.random_weights(cfg, seed=1), mx.oracle_for
    d = nx.write_model_dir(tmp_path / "m", cfg, W)
    lim = dict(dtype="bfloat16", max_tokens=4096, max_seqs=64, blocks=512)
    t = np.random.default_rng(2).integers(0, cfg["vocab"], 150).tolist()

    def free():
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    nx.open_engine(d, **lim).close()          # what a first engine loads stays loaded
    before = free()
    with nx.open_engine(d, **lim) as e:
        used = before - free()
        roomy = nx.feed_whole(e, t)
    workspace = (4096 // 64 + 64) * 16 * 128 * 130 * 4
    assert used > workspace
    hog = torch.empty(free() - (used - workspace // 2), dtype=torch.uint8, device="cuda")       # the workspace alone no longer fits
    try:
        with nx.open_engine(d, **lim) as e:
            tight = nx.feed_whole(e, t)
    finally:
        del hog
        torch.cuda.empty_cache()
    want = oracle(cfg, W).forward(t)
    a, b = np.median(nx.rel_err(tight, want)), np.median(nx.rel_err(roomy, want))
    # the other forms of the same sums, each rounded to bf16 a few times
    assert a < 0.03 and b < 0.03 and a < 1.2 * b + 1e-3, (a, b)
