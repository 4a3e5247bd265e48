"""A few rows against a wide matrix in one pass over the weights (csrc/linear_stream.cu), at the sizes where its split can go
wrong: rows that do not fill a block, fewer rows than SMs, K that is no whole number of pieces, every token block's edges."""
import pytest
import torch

from kubeai_b200 import B200Error

pytestmark = pytest.mark.gpu
# 1, 47 and 149 rows (fewer than a CTA each, one more than the SMs), 16- and 48-row blocks' edges, several blocks a CTA
SHAPES = [(1, 64), (47, 8), (149, 72), (16 * 148, 192), (16 * 148 + 1, 520), (32 * 148, 136), (32 * 148 + 8, 136), (48 * 148, 64), (48 * 148 + 3, 1000),
          (97 * 148, 72), (576, 2048), (2048, 8192)]


def operands(T, N, K, pad=0):
    g = torch.Generator(device="cuda").manual_seed(T * 131 + N * 7 + K)
    x = torch.randn(T, K + pad, generator=g, device="cuda").to(torch.bfloat16)[:, :K]
    w = torch.randn(N, K + 2 * pad, generator=g, device="cuda").mul(K ** -0.5).to(torch.bfloat16)[:, :K]
    return x, w


def close(y, want, K):
    # fp32 sums of exact products in two orders differ by at most K 2^-24 of the sum of their sizes (about sqrt(K) here: 0.8^2
    # |x||w| with |w| ~ K^-1/2), and a bf16 result by half an ulp of its own
    lim = K * 2.0 ** -24 * K ** 0.5 + (2.0 ** -8 * want.abs() if y.dtype == torch.bfloat16 else 0.0) + 1e-7
    assert ((y.double() - want).abs() <= lim).all(), ((y.double() - want).abs() - lim).max()


@pytest.mark.parametrize("N,K", SHAPES)
def test_product_matches_64_bits(N, K):
    from kubeai_b200 import ops
    for T in (1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 48):
        if T > (48 if N <= 32 * 148 else 32 if N <= 80 * 148 else 8):
            x, w = operands(T, N, K)
            with pytest.raises(B200Error):
                ops.linear_rows(x, w)
            continue
        x, w = operands(T, N, K, pad=8)
        want = x.double() @ w.double().T
        y = ops.linear_rows(x, w, dtype=torch.float32)
        close(y, want, K)
        assert torch.equal(ops.linear_rows(x, w), y.to(torch.bfloat16))     # the same sums, rounded once
        # a row's sums do not depend on what else is in the batch (within one matrix)
        assert torch.equal(ops.linear_rows(x[-1:], w, dtype=torch.float32)[0], y[-1])


def test_rows_of_other_tokens_and_of_other_blocks_stay_apart():
    """Values that are not finite reach the outputs of their own row of x or of w, and nothing is written past the sizes."""
    from kubeai_b200 import ops
    x, w = operands(9, 49 * 148 + 5, 200)
    ref = ops.linear_rows(x, w, dtype=torch.float32)
    x[3, 7], w[148, 0] = float("nan"), float("inf")
    out = torch.full((10, w.shape[0] + 8), 7.0, device="cuda")
    y = ops.linear_rows(x, w, out=out[:9, :w.shape[0]])
    assert torch.isnan(y[3]).all() and not torch.isfinite(y[:, 148]).any()
    keep = torch.ones_like(ref, dtype=torch.bool)
    keep[3], keep[:, 148] = False, False
    assert torch.equal(y[keep], ref[keep])
    assert (out[9] == 7).all() and (out[:, w.shape[0]:] == 7).all()


@pytest.mark.parametrize("N,K", [(128, 64), (2048, 192), (4096, 2048), (14336 * 2, 136)])
@pytest.mark.parametrize("act", [3, 4])
def test_pairs_match_their_plain_sums(N, K, act):
    """Gated units and silu(g) u of rows i, i + 64 of every 128: the arithmetic of the separate kernels on the plain sums."""
    from kubeai_b200 import ops
    for T in (1, 8, 13, 16, 24, 31):
        if T > (32 if N <= 80 * 148 else 8):
            continue
        x, w = operands(T, N, K)
        # the paired form deals rows out in another order but sums each of them in the same one when the split of K is the same:
        # it is, for every N
        s = ops.linear_rows(x, w).reshape(T, -1, 2, 64)
        g, u = s[:, :, 0].reshape(T, -1), s[:, :, 1].reshape(T, -1)
        if act == 4:
            assert torch.equal(ops.linear_rows(x, w, act=4), ops.silu_mul(torch.cat([g, u], 1).contiguous()))
            continue
        for lim, slope, off in ((float("inf"), 1.0, 0.0), (0.5, 1.702, 1.0)):
            gd, ud = g.double().clamp(max=lim), u.double().clamp(-lim, lim)
            want = gd * torch.sigmoid(slope * gd) * (ud + off)
            got = ops.linear_rows(x, w, act=3, p=(lim, slope, off)).double()
            assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("act", [0, 1, 2])
def test_bias_and_activations(act):
    from kubeai_b200 import ops
    x, w = operands(11, 600, 256)
    bias = torch.randn(600, device="cuda")
    z = ops.linear_rows(x, w, dtype=torch.float32).double() + bias.double()
    if act == 1:
        z = z.clamp(min=0) ** 2
    elif act == 2:
        neg = z.clamp(max=0)
        z = torch.where(z > 0, 0.8 * z * z, 1.2 * (torch.expm1(neg) - neg)) + 0.5 * z
    y = ops.linear_rows(x, w, bias=bias, act=act, p=(0.8, 1.2, 0.0), dtype=torch.float32).double()
    assert ((y - z).abs() <= 1e-5 * (1 + z.abs())).all()


@pytest.mark.parametrize("heads,kv_heads,K", [(4, 1, 256), (32, 8, 192), (12, 3, 520), (2, 2, 64)])
@pytest.mark.parametrize("T", [1, 8, 13, 32])
def test_rotated_heads_and_cache_rows_equal_the_fused_form(heads, kv_heads, K, T):
    """Small whole numbers have the same sums in every order, so both forms round the same values at the same points: the same bits, for
    tokens without a slot, positions past the table and before it, several query heads to a key head, cache rows in any order."""
    from kubeai_b200 import ops
    N, blocks = (heads + 2 * kv_heads) * 128, 5
    g = torch.Generator().manual_seed(heads * 100 + T)
    x = torch.randint(-4, 5, (T, K), generator=g).to(torch.bfloat16).cuda()
    w = torch.randint(-4, 5, (N, K), generator=g).to(torch.bfloat16).cuda()
    cs = torch.randn(40, 128, generator=g).to(torch.bfloat16).cuda()
    pos = torch.randint(0, 40, (T,), generator=g, dtype=torch.int32)
    slots = torch.randperm(blocks * 16, generator=g)[:T].to(torch.int32)
    pos[0], pos[-1] = 77, -3
    if T > 1:
        slots[T // 2] = -1
    out = torch.full((T + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    kv = torch.full((blocks, 2, kv_heads, 16, 128), 5.0, dtype=torch.bfloat16, device="cuda")
    names = dict(positions=pos.cuda(), slots=slots.cuda(), cos_sin=cs, q_heads=heads, kv_heads=kv_heads)
    ops.gemm3(x, w, epi=ops.EPI_ROPE_KV, out=out, kv_layer=kv, pairs=True, **names)
    sums = (x.float() @ w.float().T).to(torch.bfloat16).float()
    c, s = (cs[pos.clamp(0, 39).long().cuda()].float()[:, None, a:a + 64] for a in (0, 64))
    bf = lambda v: v.to(torch.bfloat16).float()
    rows = sums.reshape(T, heads + 2 * kv_heads, 128)
    a, b = rows[..., :64], rows[..., 64:]
    turned = torch.cat([bf(bf(a * c) - bf(b * s)), bf(bf(b * c) + bf(a * s))], -1)
    assert torch.equal(out[:T, :heads * 128].float().reshape(T, heads, 128), turned[:, :heads])
    assert (out[T] == 7).all() and (out[:, heads * 128:] == 7).all()
    want = torch.full_like(kv, 5.0)
    for t in range(T):
        if slots[t] >= 0:
            want[slots[t] // 16, 0, :, slots[t] % 16] = turned[t, heads:heads + kv_heads].to(torch.bfloat16)
            want[slots[t] // 16, 1, :, slots[t] % 16] = rows[t, heads + kv_heads:].to(torch.bfloat16)
    assert torch.equal(kv, want)
    if N % 256 == 0 and K % 64 == 0:      # sizes of the fused form
        fused, kv2 = torch.zeros(T, N, dtype=torch.bfloat16, device="cuda"), torch.full_like(kv, 5.0)
        ops.gemm3(x, w, epi=ops.EPI_ROPE_KV, out=fused, kv_layer=kv2, **names)
        assert torch.equal(fused[:, :heads * 128], out[:T, :heads * 128]) and torch.equal(kv2, kv)
