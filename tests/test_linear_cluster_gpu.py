"""Products of some tens to a few hundred rows with K cut over clusters (csrc/linear_cluster.cu): rows of W that do not fill a
cluster, K that does not fill a stage or a CTA's share, both sides of every line of its choice of shape."""
import pytest
import torch

from kubeai_b200 import B200Error

pytestmark = pytest.mark.gpu


def operands(T, N, K, pad=0):
    g = torch.Generator(device="cuda").manual_seed(T * 131 + N * 7 + K)
    x = torch.randn(T, K + pad, generator=g, device="cuda").to(torch.bfloat16)[:, :K]
    w = torch.randn(N, K + 2 * pad, generator=g, device="cuda").mul(K ** -0.5).to(torch.bfloat16)[:, :K]
    return x, w


@pytest.mark.parametrize("N,K", [(1024, 512), (1030, 520), (2048, 1000), (2047, 2048), (2112, 4088), (2112, 4096), (2049, 4104), (2048, 8192), (2113, 512), (3072, 1024),
                                 (3168, 648), (1027, 6000)])
def test_product_matches_64_bits(N, K):
    from kubeai_b200 import ops
    for T in (49, 64, 65, 96, 97, 128, 129, 160, 161, 255, 256):
        if N > 2112 and T > 128:
            x, w = operands(T, N, K)
            with pytest.raises(B200Error):
                ops.linear_rows(x, w)
            continue
        x, w = operands(T, N, K, pad=8)
        want = x.double() @ w.double().T
        out = torch.full((T + 1, N + 12), 7.0, device="cuda")
        y = ops.linear_rows(x, w, out=out[:T, :N])
        # fp32 sums of exact products in two orders: at most K 2^-24 of the sum of their sizes
        assert ((y.double() - want).abs() <= K * 2.0 ** -24 * K ** 0.5 + 1e-7).all()
        assert (out[T] == 7).all() and (out[:, N:] == 7).all()
        assert torch.equal(ops.linear_rows(x, w), y.to(torch.bfloat16))
        for _ in range(3):
            assert torch.equal(ops.linear_rows(x, w, dtype=torch.float32), y)     # the parts are added in one order


@pytest.mark.parametrize("rank", [1024, 1100])
def test_the_one_head_of_a_latent_layer(tmp_path, rank):
    """A latent layer of one head has its per-head products here; their waits are reported like the others'."""
    import numpy as np

    import soselix_util as sx
    from nomanex_util import feed_portions, open_engine, rel_err, write_model_dir
    cfg = sx.make_config([sx.latent(heads=1, dim=64, rot_dim=8, vdim=16, kv_rank=rank, q_rank=32, mlp=None)], width=64)
    W = sx.random_weights(cfg, seed=rank)
    d = write_model_dir(tmp_path / "m", cfg, W)
    t = np.random.default_rng(rank).integers(0, cfg["vocab"], 1 + 64 + 130).tolist()
    with open_engine(d, dtype="bfloat16") as e:
        r = rel_err(feed_portions(e, t, [1, 64, 130]), sx.oracle_for(cfg, W).forward(t))
    # six operators' outputs rounded to 2^-9 of their size each, on a width of 64
    assert np.median(r) < 0.03 and r.max() < 0.2, (np.median(r), r.max())


@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("T", [50, 130])
def test_bias_and_activations(act, T):
    from kubeai_b200 import ops
    x, w = operands(T, 1500, 768)
    bias = torch.randn(1500, device="cuda")
    z = ops.linear_rows(x, w, dtype=torch.float32).double() + bias.double()
    if act == 1:
        z = z.clamp(min=0) ** 2
    elif act == 2:
        neg = z.clamp(max=0)
        z = torch.where(z > 0, 0.8 * z * z, 1.2 * (torch.expm1(neg) - neg)) + 0.5 * z
    y = ops.linear_rows(x, w, bias=bias, act=act, p=(0.8, 1.2, 0.0), dtype=torch.float32).double()
    assert ((y - z).abs() <= 1e-5 * (1 + z.abs())).all()


def test_rows_stay_apart():
    from kubeai_b200 import ops
    x, w = operands(70, 2048, 1024)
    ref = ops.linear_rows(x, w, dtype=torch.float32)
    x[33, 7], w[65, 0] = float("nan"), float("inf")
    y = ops.linear_rows(x, w, dtype=torch.float32)
    assert torch.isnan(y[33]).all() and not torch.isfinite(y[:, 65]).any()
    keep = torch.ones_like(ref, dtype=torch.bool)
    keep[33], keep[:, 65] = False, False
    assert torch.equal(y[keep], ref[keep])
