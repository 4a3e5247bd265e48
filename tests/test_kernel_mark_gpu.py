"""A kernel that gave up waiting leaves a mark.  The step it belongs to fails, not the one after it; an operation that returns
before its kernel has run is reported by the next.  (The mark is set by hand: no kernel is made to wait in vain.)"""
import numpy as np
import pytest
import torch

import soselix_util as sx

pytestmark = pytest.mark.gpu


def design(tmp_path):
    cfg = sx.make_config([sx.latent(), sx.hgrn2()])
    return sx.open_engine(sx.write_model_dir(tmp_path / "m", cfg, sx.random_weights(cfg, seed=1)), dtype="bfloat16")


def llama(tmp_path):
    from kubeai_b200.engine import Engine, mini_config
    return Engine(mini_config())


@pytest.mark.parametrize("make", [design, llama])
def test_a_fed_step_that_ends_with_the_mark_set_fails(tmp_path, make):
    with make(tmp_path) as e:
        assert e._l.b200_engine_kernel_mark(e._h, -1) == 0
        r = e.feed_open()
        e.feed_step([(r, [1, 2, 3], [2])])
        steps = e.stats().steps
        assert e._l.b200_engine_kernel_mark(e._h, 1) == 0
        with pytest.raises(RuntimeError, match="wait inside a kernel"):
            e.feed_step([(r, [4], [0])])
        assert e._l.b200_engine_is_failed(e._h) == 1 and e.stats().steps == steps
        with pytest.raises(RuntimeError):          # nothing can build on that step
            e.feed_step([(r, [4], [0])])
        with pytest.raises(RuntimeError):
            e.submit([1, 2, 3], max_tokens=2)


@pytest.mark.parametrize("make", [design, llama])
def test_a_fed_step_that_fails_leaves_the_callers_memory_as_it_was(tmp_path, make):
    import ctypes as C
    from kubeai_b200._lib import FeedEntry
    with make(tmp_path) as e:
        rows = 16
        out = np.full((rows, e.cfg.vocab), 7.0, dtype=np.float32)
        tokens, want = (C.c_int32 * rows)(*(i % 30 for i in range(rows))), (C.c_int32 * rows)(*range(rows))
        entry = (FeedEntry * 1)()
        entry[0].req_id = e.feed_open()
        entry[0].n_tokens = entry[0].n_want = rows
        entry[0].tokens, entry[0].want = tokens, want
        e._l.b200_engine_kernel_mark(e._h, 1)
        assert e._l.b200_feed_step(e._h, entry, 1, out.ctypes.data_as(C.POINTER(C.c_float)), out.size) < 0
        assert b"wait inside a kernel" in e._l.b200_last_error() and (out == 7.0).all()


@pytest.mark.parametrize("make", [design, llama])
def test_a_scheduled_step_that_ends_with_the_mark_set_hands_out_no_token(tmp_path, make):
    with make(tmp_path) as e:
        r = e.submit([5, 6, 7], max_tokens=4)
        e._l.b200_engine_kernel_mark(e._h, 1)
        assert e._l.b200_engine_step(e._h, None) < 0
        assert e.poll(r).tokens == [] and e._l.b200_engine_is_failed(e._h) == 1


def test_a_product_is_reported_by_the_next_one(tmp_path):
    from kubeai_b200 import ops
    x, w = torch.randn(8, 256, device="cuda").to(torch.bfloat16), torch.randn(64, 256, device="cuda").to(torch.bfloat16)
    want = ops.gemm(x, w)
    assert ops.lib().b200_op_kernel_mark(1) == 0
    with pytest.raises(RuntimeError, match="earlier product"):
        ops.gemm(x, w)
    assert ops.lib().b200_op_kernel_mark(-1) == 0
    assert torch.equal(ops.gemm(x, w), want)
    assert np.isfinite(want.float().cpu().numpy()).all()
