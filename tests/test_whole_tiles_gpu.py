"""The whole-tile product (csrc/gemm_grouped.cu): every size of its row tiles and operand boxes, K whole and in parts, and the
expert form behind a model, against 64-bit products and against the tile kernel it replaces."""
import math

import numpy as np
import pytest
import torch

import soselix_util as sx
from mulenex_util import attention, bf16_round, dense, layer, make_config, moe, mlstm, open_engine, feed_whole, random_weights, rel_err, write_model_dir, oracle_for

pytestmark = pytest.mark.gpu


def operands(T, N, K, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") / math.sqrt(K)).to(torch.bfloat16)
    return x, w


@pytest.mark.parametrize("T,N,K", [
    (1, 8, 8), (1, 4096, 4096), (16, 264, 72), (17, 2048, 2048), (32, 2048, 8192), (33, 1032, 4096),      # boxes of 16 and 32 rows, K in parts
    (64, 256, 16384), (65, 2048, 2048), (128, 4096, 14336), (129, 2048, 4104), (255, 512, 2048), (256, 4096, 4096),   # 64 and 128; K no whole steps
    (257, 4096, 14336), (300, 2048, 8192), (511, 264, 1032), (513, 2048, 2048),                       # two and three row tiles
    (1000, 6144, 4096), (1999, 4096, 2048), (2048, 8192, 1024),                                          # several waves
])
def test_product_against_64_bits_and_repeatable(T, N, K):
    from kubeai_b200 import ops
    x, w = operands(T, N, K)
    got = ops.gemm(x, w)
    again = ops.gemm(x, w)          # counters are zero again, the parts are added in their order whoever comes last
    assert torch.equal(got, again)
    want = x.double() @ w.double().T
    # one rounding to bf16 (8 significant bits: half a last place is at most 2^-8 of the value) and at most K + 16 fp32
    # additions (2^-24 of the sum of magnitudes each)
    bound = 2.0 ** -8 * want.abs() + (K + 16) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert ((got.double() - want).abs() <= 1.01 * bound + 1e-30).all()


@pytest.mark.parametrize("T", [63, 64, 65, 96, 97, 128, 129, 256, 257, 320, 321])
@pytest.mark.parametrize("N,K", [(256, 3072), (512, 8200), (768, 2048), (1024, 4104), (1536, 3080), (1544, 3072)])
def test_few_weight_tiles_and_a_long_k(T, N, K):
    """Both sides of the lines between the whole tiles and the stream-K kernel: the same bound."""
    from kubeai_b200 import ops
    x, w = operands(T, N, K, seed=2)
    got, again = ops.gemm(x, w), ops.gemm(x, w)
    assert torch.equal(got, again)
    want = x.double() @ w.double().T
    bound = 2.0 ** -8 * want.abs() + (K + 16) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert ((got.double() - want).abs() <= 1.01 * bound + 1e-30).all()


def test_infinities_and_nan_stay_in_their_rows():
    from kubeai_b200 import ops
    x, w = operands(40, 512, 8192, seed=3)
    x[3, 100], x[7, 5000] = float("nan"), float("inf")
    got = ops.gemm(x, w)
    assert torch.isnan(got[3]).all() and not torch.isfinite(got[7]).any()
    rest = [i for i in range(40) if i not in (3, 7)]
    assert torch.isfinite(got[rest]).all()


@pytest.mark.parametrize("ff,shared", [(64, 64), (24, 40), (128, None)])
@pytest.mark.parametrize("T", [33, 64, 65, 129, 255, 256, 300])
def test_experts_agree_with_the_tile_kernel(tmp_path, monkeypatch, ff, shared, T):
    """Interleaved and stacked gate and up rows, fp32 outputs below 256 tokens, every operand box."""
    layers = [layer(attention(heads=2, kv_heads=1, dim=16, vdim=16), mlp=moe(experts=5, top=2, ff=ff, shared=shared)),
              layer(mlstm(heads=2, dim=16, vdim=16), mlp=moe(experts=3, top=3, ff=ff, shared=shared))]
    cfg = make_config(layers, width=64)
    W = random_weights(cfg, seed=5)
    d = write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(T).integers(0, cfg["vocab"], T).tolist()
    with open_engine(d, dtype="bfloat16") as e:
        new = feed_whole(e, t)
    monkeypatch.setenv("B200_MX_MOE_TC_MIN_T", "100000")
    with open_engine(d, dtype="bfloat16") as e:
        old = feed_whole(e, t)
    want = oracle_for(cfg, W).forward(t)
    # both round every projection to bf16, so a row's distance to the oracle is a few times 2^-8; rows whose routing is close
    # to a tie may take another expert
    assert np.median(rel_err(new, want)) < 0.03 and np.median(rel_err(new, old.astype(np.float64))) < 0.02
    assert np.median(rel_err(new, want)) < 1.3 * np.median(rel_err(old, want)) + 1e-3


def picks(rng, rows, cols):
    """One power of two per row: every product with it is exact, whatever the order of the sum."""
    m = np.zeros((rows, cols), dtype=np.float32)
    m[np.arange(rows), rng.integers(0, cols, rows)] = 2.0 ** rng.integers(-1, 4, rows) * rng.choice([-1.0, 1.0], rows)
    return m


@pytest.mark.parametrize("T", [40, 250])
def test_gated_unit_in_the_epilogue_is_the_one_of_its_own_kernel(tmp_path, monkeypatch, T):
    """Same accurate exponential and quotient: where the sums are exact, so are the two forms equal, bit for bit."""
    cfg = make_config([layer(attention(heads=2, kv_heads=1, dim=16, vdim=16), mlp=moe(experts=4, top=2, ff=512, shared=None))], width=512)
    W, rng = random_weights(cfg, seed=6), np.random.default_rng(7)
    for e in range(4):
        W["l0.mlp.e%d.gate" % e], W["l0.mlp.e%d.up" % e], W["l0.mlp.e%d.down" % e] = (picks(rng, 512, 512) for _ in range(3))
    d = write_model_dir(tmp_path / "m", cfg, W)
    t = rng.integers(0, cfg["vocab"], T).tolist()
    out = []
    for least in ("1", "100000"):            # tokens from which the experts take the grouped product
        monkeypatch.setenv("B200_MX_MOE_TC_MIN_T", least)
        with open_engine(d, dtype="bfloat16") as e:
            out.append(feed_whole(e, t))
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("T", [17, 64, 130, 300])
def test_split_products_with_an_epilogue(tmp_path, monkeypatch, T):
    """Few weight tiles and a long K: the last part adds the others and goes on to the bias and squared ReLU, the gated unit of a
    shared expert, or the bias and xIELU."""
    monkeypatch.setenv("B200_SX_FEW_ROWS", "1")
    mxc = make_config([layer(attention(heads=2, kv_heads=1, dim=16, vdim=16), mlp=dense(ff=264)),
                       layer(attention(heads=2, kv_heads=1, dim=16, vdim=16, v_mix=False), mlp=moe(experts=2, top=1, ff=64, shared=192))], width=2048)
    sxc = sx.make_config([sx.latent(), dict(sx.hgrn2(), mlp=sx.dense(ff=520))], width=2048)
    for name, cfg, weights, oracle, knob in (("mx", mxc, random_weights, oracle_for, "B200_MX_TC"), ("sx", sxc, sx.random_weights, sx.oracle_for, "B200_SX_TC")):
        W = weights(cfg, seed=T)
        d = write_model_dir(tmp_path / name, cfg, W)
        t = np.random.default_rng(T).integers(0, cfg["vocab"], T).tolist()
        out = []
        for on in ("1", "0"):                # "0": unsplit tile kernels of linear.cu and the epilogues' own kernels
            monkeypatch.setenv(knob, on)
            with open_engine(d, dtype="bfloat16") as e:
                out.append(rel_err(feed_whole(e, t), oracle(cfg, W).forward(t)))
        # the fused form rounds once less per product; otherwise the same roundings
        assert np.median(out[0]) < 0.03 and np.median(out[0]) < 1.1 * np.median(out[1]) + 2.0 ** -11, (name, np.median(out[0]), np.median(out[1]))
        assert out[0].max() < 3 * out[1].max() + 2.0 ** -8, (name, out[0].max(), out[1].max())


@pytest.mark.parametrize("T", [9, 16, 17, 33, 64, 65, 96, 112, 113])
@pytest.mark.parametrize("I,K", [(128, 64), (1024, 512), (3584, 1024), (14336, 4096)])
def test_gate_and_up_of_a_step(T, I, K):
    """Both sides of the lines between the passes over the weights, whole tiles and the kernel of a decode step's pairs."""
    from kubeai_b200 import ops
    x, w = operands(T, 2 * I, K, seed=4)
    got, again = ops.gemm3(x, w, epi=ops.EPI_SILU)[0], ops.gemm3(x, w, epi=ops.EPI_SILU)[0]
    assert torch.equal(got, again)
    gu = x.double() @ w.double().T
    mag = (K + 16) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    (g, u), (dg, du) = ((t.reshape(T, I // 64, 2, 64).transpose(1, 2).reshape(T, 2, I).unbind(1)) for t in (gu, 2.0 ** -8 * gu.abs() + mag))
    s = g * torch.sigmoid(g)
    # g and u rounded to bf16, silu(g) (its slope is at most 1.1) rounded again, the product rounded again
    ds = 1.1 * dg + 2.0 ** -8 * (s.abs() + 1.1 * dg)
    bound = ds * (u.abs() + du) + s.abs() * du
    bound = bound + 2.0 ** -8 * ((s * u).abs() + bound)
    assert ((got.double() - s * u).abs() <= 1.01 * bound + 1e-30).all()
