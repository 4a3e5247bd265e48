"""Steps of few tokens of the built-in kernel sequence on the one-pass products (csrc/linear_stream.cu) against the fused form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [dict(hidden=1024, q_heads=8, kv_heads=2, intermediate=3584),
                                   dict(hidden=4096, q_heads=32, kv_heads=8, intermediate=14336)])
@pytest.mark.parametrize("T", [1, 9, 17, 24, 25, 32, 33, 40, 48, 49])
def test_few_token_steps_agree_with_the_fused_form(shape, T, monkeypatch):
    """Prompts of T tokens in one step, then T decode steps of a few sequences: the logits of both forms differ by roundings."""
    from kubeai_b200.engine import Engine, mini_config
    out = []
    for knob in ("1", "0"):
        monkeypatch.setenv("B200_FEW_ROWS", knob)
        with Engine(mini_config(max_num_seqs=64, max_batched_tokens=128, max_model_len=128, num_kv_blocks=64, num_layers=2, **shape)) as e:
            rng = np.random.default_rng(T)
            n = [T - T // 3, T // 3] if T > 2 else [T]
            ids = [e.feed_open() for _ in n]
            got = [e.feed_step([(r, rng.integers(0, 512, k), list(range(k))) for r, k in zip(ids, n)])]
            for _ in range(3):
                got.append(e.feed_step([(r, rng.integers(0, 512, 1), [0]) for r in ids]))
            out.append(np.concatenate([np.concatenate([np.asarray(v, dtype=np.float64).reshape(-1, 512) for v in s]) for s in got]))
    a, b = out
    # both forms round at the same points; sums in another order move an output of every product by at most one bf16 ulp, which
    # two layers carry on: 2^-8 of a row's size for each of the eight products and the head, random signs
    rel = np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)
    assert rel.max() < 9 ** 0.5 * 2.0 ** -8 * 2, rel.max()


@pytest.mark.parametrize("T", [9, 33, 64, 65, 128])
def test_gate_and_up_with_few_tiles_left_for_a_second_round(T, monkeypatch):
    """The other projections take whole tiles, gate and up the pairs of the fused form (rules::gate_up_tiles): against the fused form alone."""
    import ctypes as C
    import torch
    from kubeai_b200.engine import Engine, mini_config
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    inter = (pairs + 2) * 128
    out = []
    for knob in ("1", "0"):
        monkeypatch.setenv("B200_FEW_ROWS", knob)
        with Engine(mini_config(max_num_seqs=4, max_batched_tokens=128, max_model_len=256, num_kv_blocks=64, hidden=3072, q_heads=24, kv_heads=6, intermediate=inter)) as e:
            assert e._l.b200_rule_query(13, (C.c_int32 * 3)(2 * inter, 3072, pairs), 3) == 0
            r = e.feed_open()
            out.append(np.asarray(e.feed_step([(r, np.random.default_rng(T).integers(0, 512, T), [0, T // 2, T - 1])]), dtype=np.float64))
    a, b = out
    # as above: eight products and the head, each an ulp at most
    rel = np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)
    assert rel.max() < 9 ** 0.5 * 2.0 ** -8 * 2, rel.max()
