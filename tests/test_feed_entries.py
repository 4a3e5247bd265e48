"""Fed steps: the entries as they reach the C call, whatever the caller's sequences are made of, and the logits that come back
in more than one part."""
import numpy as np
import pytest

from kubeai_b200 import engine as E


class Recorder:
    def b200_feed_step(self, h, arr, n, out, size):
        self.seen = [(arr[i].req_id, arr[i].tokens[:arr[i].n_tokens], arr[i].want[:arr[i].n_want] if arr[i].want else None) for i in range(n)]
        return 0


def fed(entries):
    e = E.Engine.__new__(E.Engine)
    e._l, e._h, e.cfg = Recorder(), None, E.Config(vocab=7)
    out = e.feed_step(entries)
    assert out.dtype == np.float32 and out.shape == (sum(len(w) for _, _, w in entries), 7)
    return e._l.seen


@pytest.mark.parametrize("entries,want", [
    ([(3, [1, 2, 3], [0, 2])], [(3, [1, 2, 3], [0, 2])]),
    ([(1, np.arange(8)[::2], []), (2, (7,), np.array([0]))], [(1, [0, 2, 4, 6], None), (2, [7], [0])]),
    ([(2 ** 63 + 5, np.array([4], dtype=np.uint8), [0]), (9, [], [])], [(2 ** 63 + 5, [4], [0]), (9, [], None)]),
    ([(1, np.array([[5, 6], [7, 8]]), []), (np.uint64(2), [1], [0])], [(1, [5, 6], None), (2, [1], [0])]),
    ([], []),
])
def test_entries(entries, want):
    assert fed(entries) == want


@pytest.mark.parametrize("entries,error", [([(1.5, [1], [])], TypeError), ([(1, [2 ** 40], [])], OverflowError), ([(1, [1])], ValueError),
                                           ([(1, [1], []), (1, [1], [], 0)], ValueError), ([(1, ["a"], [])], ValueError)])
def test_refused_entries(entries, error):
    with pytest.raises(error):
        fed(entries)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 64, 65, 97, 128])
def test_logits_in_parts(rows):
    """32 rows of 32768 are one part; from the third part on a half of the staging memory is used again."""
    cfg = E.default_config(num_layers=1, hidden=512, q_heads=8, kv_heads=2, intermediate=1024, vocab=32768, manual_step=1, max_num_seqs=128,
                           max_batched_tokens=256, max_model_len=64, num_kv_blocks=512)
    with E.Engine(cfg) as e:
        e.set_keep_logits(True)
        ids = [e.feed_open() for _ in range(rows)]
        got = e.feed_step([(r, [i + 1, 2 * i + 1], [1]) for i, r in enumerate(ids)])
        assert np.isfinite(got).all() and got.std(axis=1).min() > 0
        np.testing.assert_array_equal(got, e.read_logits(rows))


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 64])
def test_logits_of_a_design_around_the_staging_limit(tmp_path, rows):
    """32 rows of 32768 fp32 logits are staged, 33 go to the caller's memory at once: the same numbers row by row."""
    import soselix_util as sx
    cfg = sx.make_config([sx.hgrn2(mlp=None)], vocab=32768)
    W = sx.random_weights(cfg, seed=2)
    with sx.open_engine(sx.write_model_dir(tmp_path / "m", cfg, W), dtype="bfloat16", max_tokens=128) as e:
        t = np.random.default_rng(1).integers(0, 32768, rows).tolist()
        r = e.feed_open()
        got = e.feed_step([(r, t, list(range(rows)))])
        e.feed_close(r)
        parts = []
        for lo in range(0, rows, 20):        # the same step, twenty positions of it at a time
            r = e.feed_open()
            parts.append(e.feed_step([(r, t, list(range(lo, min(rows, lo + 20))))]))
            e.feed_close(r)
    assert np.isfinite(got).all() and got.std(axis=1).min() > 0
    # other numbers of rows take other product kernels: the same sums in another order
    np.testing.assert_allclose(got, np.concatenate(parts), rtol=0, atol=2.0 ** -20 * 64 * np.abs(got).max())


def test_arrays_and_lists_give_the_same_entries():
    """int32 vectors go through the native packing, everything else through numpy: the C call sees the same."""
    rng = np.random.default_rng(5)
    toks = [rng.integers(0, 7, n).astype(np.int32) for n in (1, 3, 17, 2)]
    wants = [np.array(w, dtype=np.int32) for w in ([], [2], [0, 16], [])]
    rids = [1, 2 ** 64 - 1, 7, 2 ** 63]
    plain = [(r, t.tolist(), w.tolist()) for r, t, w in zip(rids, toks, wants)]
    want = [(r, t, w or None) for r, t, w in plain]
    assert fed(list(zip(rids, toks, wants))) == fed(plain) == fed(tuple(zip(rids, toks, wants))) == want
    # one entry that is not such a vector sends the whole step the other way: strides, byte order, width, a second dimension, an id that is no int
    for odd in (np.arange(6, dtype=np.int32)[::2], toks[1].astype(">i4"), toks[1].astype(np.int64), toks[1]):
        assert fed([(5, toks[0], wants[0]), (np.int64(6), odd, wants[1])]) == [(5, toks[0].tolist(), None), (6, odd.tolist(), [2])]
    assert fed([(5, np.ones((3, 1), dtype=np.int32), wants[1])]) == [(5, [1, 1, 1], [2])]


def helper():
    """The native packing, where the headers it is built with are there."""
    from kubeai_b200 import _build
    if not _build._feed_flags():
        pytest.skip("no headers of Python or numpy")
    from kubeai_b200 import _feed
    assert E._pack is _feed.pack
    return _feed


def test_the_native_packing_serves_int32_vectors_and_nothing_else():
    pack = helper().pack
    t, w = np.array([1, 2, 3], dtype=np.int32), np.array([0, 2], dtype=np.int32)
    buf, rows = pack([(7, t, w), (8, t[:1], w[:0])])
    assert isinstance(buf, bytearray) and rows == 2
    for odd in ([(7, [1, 2, 3], w)], [(7, t, [0, 2])], ((7, t, w),), [[7, t, w]], [(np.int64(7), t, w)], [(True, t, w)], [(7, t.astype(np.int64), w)], [(7, t[::2], w)],
                [(7, t.astype(">i4"), w)], [(7, t.reshape(1, 3), w)], [(7, t)], [(7, t, w), (8, t, w, w)], []):
        assert pack(odd) is None, odd


def test_the_native_packing_belongs_to_one_interpreter():
    import sysconfig
    from kubeai_b200 import _build
    name = helper().__file__.rsplit("/", 1)[-1]
    assert name == "_feed" + sysconfig.get_config_var("EXT_SUFFIX") != "_feed.so" and _build.FEED.name == name


def test_another_numpy_or_interpreter_is_another_build(monkeypatch):
    import sys
    from kubeai_b200 import _build
    a = _build._feed_digest(["-Ix"])
    assert a == _build._feed_digest(["-Ix"]) != _build._feed_digest(["-Iy"])
    with monkeypatch.context() as m:
        m.setattr(np, "__version__", "0.1")
        assert _build._feed_digest(["-Ix"]) != a
    with monkeypatch.context() as m:
        m.setattr(sys, "version", "2.7")
        assert _build._feed_digest(["-Ix"]) != a


def test_a_compiler_that_fails_costs_the_helper_and_no_more(monkeypatch, tmp_path, capsys):
    from kubeai_b200 import _build
    monkeypatch.setattr(_build, "OBJ", tmp_path / "obj")
    monkeypatch.setattr(_build, "FEED", tmp_path / "_feed.x.so")
    monkeypatch.setattr(_build, "_feed_flags", lambda: ["-no-such-flag"])
    (tmp_path / "_feed.so").write_bytes(b"any interpreter would take this")
    (tmp_path / "_feed.x.so").write_bytes(b"of another source")
    assert _build.build_feed() is False and "formed by numpy" in capsys.readouterr().err
    assert not list(tmp_path.glob("*.so"))
    monkeypatch.setattr(_build, "_feed_flags", lambda: [])
    assert _build.build_feed() is False
