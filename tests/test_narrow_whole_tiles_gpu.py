"""Llama steps of more than 128 tokens on the whole-tile product where neither gate_up nor down fills the device: both are
resident beside the norms around them, so nothing but the launch order's own waits keeps a step's kernels apart."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from oracle.llama_oracle import LlamaOracle
from oracle.weights import ModelCfg, make_weights

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent
LENS = [129, 150, 200, 256, 300, 512]
SHAPES = {"2816": dict(hidden=1024, q_heads=8, kv_heads=2, intermediate=2816), "4096": dict(hidden=1536, q_heads=12, kv_heads=3, intermediate=4096)}


def wanted(n):
    return sorted({0, n - 1, *range(3, n, max(1, n // 40))})


def logits(shape):
    from kubeai_b200.engine import Engine, mini_config
    out = {}
    with Engine(mini_config(num_layers=4, max_model_len=512, max_batched_tokens=512, max_num_seqs=64, num_kv_blocks=256, **SHAPES[shape])) as e:
        for n in LENS:
            t = np.random.default_rng(n).integers(0, 512, n).tolist()
            for again in range(3):
                r = e.feed_open()
                out[f"{n}.{again}"] = e.feed_step([(r, t, wanted(n))])
                e.feed_close(r)
    return out


@pytest.mark.parametrize("shape", list(SHAPES))
def test_steps_follow_the_oracle_and_need_no_launch_order_to_be_right(tmp_path, shape):
    got = logits(shape)
    # every kernel launched only when the one in front of it has ended: the same numbers, bit for bit
    code = f"import numpy as np; from test_narrow_whole_tiles_gpu import logits; np.savez({str(tmp_path / 'plain.npz')!r}, **logits({shape!r}))"
    env = dict(os.environ, B200_PDL="0", PYTHONPATH=f"{ROOT}:{ROOT / 'tests'}")
    subprocess.run([sys.executable, "-c", code], env=env, cwd=ROOT, check=True, timeout=300)
    plain = np.load(tmp_path / "plain.npz")
    for k, v in got.items():
        np.testing.assert_array_equal(v, plain[k], err_msg=k)
    ocfg = ModelCfg(num_layers=4, max_model_len=512, **SHAPES[shape])
    oracle = LlamaOracle(ocfg, make_weights(ocfg))
    for n in LENS:
        want = oracle.forward(np.random.default_rng(n).integers(0, 512, n).tolist())[0].numpy()[wanted(n)]
        err = got[f"{n}.0"] - want
        # engine and oracle round at the same points, seven a layer, and differ where another order of a sum turns a rounding: each
        # rounding that turns is 2^-8 of a value at most, of 2^-8 / sqrt(3) root mean square, and 28 of them add in quadrature
        rms = np.sqrt((err ** 2).mean(axis=-1) / (want ** 2).mean())
        assert np.median(rms) < np.sqrt(28 / 3) * 2.0 ** -8 and rms.max() < 4 * np.sqrt(28 / 3) * 2.0 ** -8, (n, np.median(rms), rms.max())
