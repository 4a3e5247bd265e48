"""Decode attention over contexts of one tile (csrc/attention.cu, one tile a CTA): at the edges of its pages, against the kernel with several tiles in flight, which a
wider block table asks for, bit by bit, and against 64 bits; in parts too.  Pages that are not there are not loaded: what lay in shared memory before must not matter."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HEADS, KV_HEADS, D = 8, 2, 128
CONTEXTS = [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64]


def cache(contexts, seed, fill=None):
    g = torch.Generator(device="cuda").manual_seed(seed)
    pages = sum(-(-c // 16) for c in contexts) + 1
    kv = torch.randn(pages, 2, KV_HEADS, 16, D, generator=g, device="cuda").to(torch.bfloat16)
    if fill is not None:
        kv.fill_(fill)
    order = torch.randperm(pages - 1, generator=g, device="cuda") + 1
    table, at = torch.zeros(len(contexts), 4, dtype=torch.int32, device="cuda"), 0
    for i, c in enumerate(contexts):
        n = -(-c // 16)
        table[i, :n] = order[at:at + n].to(torch.int32)
        at += n
        kv[table[i, n - 1].long(), :, :, (c - 1) % 16 + 1:] = 0        # behind the last token nothing has been written
    q = torch.randn(len(contexts), (HEADS + 2 * KV_HEADS) * D, generator=g, device="cuda").to(torch.bfloat16)
    work = torch.tensor([[i, 1, c - 1, i] for i, c in sorted(enumerate(contexts), key=lambda x: -x[1])], dtype=torch.int32, device="cuda")
    return q, kv, table, work


@pytest.mark.parametrize("contexts", [[c] for c in CONTEXTS] + [CONTEXTS, CONTEXTS * 20])
@pytest.mark.parametrize("split", [None, 1, 2, 5])
def test_one_tile_a_cta(contexts, split):
    from kubeai_b200 import ops
    run = lambda q, kv, table, work: ops.paged_attn(q, kv, table, work, HEADS, KV_HEADS, decode=True, **({} if split is None else {"split": split}))
    wide = lambda t: torch.cat([t, t[:, :1]], 1).contiguous()
    q, kv, table, work = cache(contexts, seed=len(contexts))
    poison = cache([64] * 300, seed=1, fill=float("nan"))
    run(*poison)
    got = run(q, kv, table, work)
    run(*poison)
    again = run(q, kv, table, work)
    several = run(q, kv, wide(table), work)
    assert torch.isfinite(got.float()).all() and torch.equal(got, again) and torch.equal(got, several)
    for i, c in enumerate(contexts[:40]):
        rows = kv[table[i].long()].permute(1, 2, 0, 3, 4).reshape(2, KV_HEADS, 64, D)[:, :, :c].double()
        qd = q[i, :HEADS * D].reshape(KV_HEADS, HEADS // KV_HEADS, D).double()
        s = torch.einsum("khd,kld->khl", qd, rows[0]) * D ** -0.5
        want = torch.einsum("khl,kld->khd", s.softmax(-1), rows[1]).reshape(-1)
        # the weights rounded to bf16 (their sum is not), the output rounded once more
        assert ((got[i, :HEADS * D].double() - want).abs() <= 2 * 2.0 ** -8 * rows[1].abs().max()).all()


def test_one_token_more_takes_the_other_kernel():
    from kubeai_b200 import ops
    q, kv, table, work = cache([64, 64], seed=3)
    longer = torch.cat([table, torch.zeros_like(table[:, :1])], 1).contiguous()
    w65 = work.clone()
    w65[:, 2] = 64
    got = ops.paged_attn(q, kv, longer, w65, HEADS, KV_HEADS, decode=True)
    rows = kv[longer[0].long()].permute(1, 2, 0, 3, 4).reshape(2, KV_HEADS, 80, D)[:, :, :65].double()
    s = torch.einsum("khd,kld->khl", q[0, :HEADS * D].reshape(KV_HEADS, HEADS // KV_HEADS, D).double(), rows[0]) * D ** -0.5
    want = torch.einsum("khl,kld->khd", s.softmax(-1), rows[1]).reshape(-1)
    assert ((got[0, :HEADS * D].double() - want).abs() <= 2 * 2.0 ** -8 * rows[1].abs().max()).all()
