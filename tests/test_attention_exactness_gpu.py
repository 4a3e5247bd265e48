"""Both kernels of prompt attention (csrc/attention_tc.cu over pages, csrc/prompt_attention.cu over whole prompts) against the same steps in 64 bits: weights
relative to the largest score met so far, which makes the row's largest weight exactly 1, rounded to bf16, and the output rounded to bf16.  Those two
roundings are all that a result may be off by; a weight that is relative to anything else costs a row with few large scores a rounding more."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def bf(t):
    return t.to(torch.bfloat16)


def attention(q, k, v, scale, rounded_sum, cap=0.0, window=None, sink=None):
    """q [n, H, d], k [n, Hk, d], v [n, Hk, 128] in 64 bits -> the exact result and the one with the two roundings."""
    n, heads = q.shape[:2]
    tiles = -(-n // 64)
    i = torch.arange(n, device=DEV)
    hidden = i[None] > i[:, None]
    if window:
        hidden |= i[None] <= i[:, None] - window
    exact, rounded = torch.empty(n, heads, 128, dtype=torch.float64, device=DEV), torch.empty(n, heads, 128, dtype=torch.float64, device=DEV)
    for h in range(heads):
        kv = h * k.shape[1] // heads
        s = q[:, h] @ k[:, kv].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s.masked_fill_(hidden, -math.inf)
        top = s.amax(1, keepdim=True)
        behind = torch.exp(sink[h].double() - top) if sink is not None else torch.zeros_like(top)
        w = torch.exp(s - top)
        exact[:, h] = w @ v[:, kv] / (w.sum(1, keepdim=True) + behind)
        pad = torch.nn.functional.pad(s, (0, 64 * tiles - n), value=-math.inf).reshape(n, tiles, 64)
        ref = pad.amax(2).cummax(1).values.clamp_min(-1e300)                # the largest score up to each tile of 64 keys
        p = torch.exp(pad - ref[:, :, None])
        back = torch.exp(ref - top)[:, :, None]
        pr = bf(p.float()).double()
        total = ((pr if rounded_sum else p) * back).sum((1, 2))[:, None] + behind
        rounded[:, h] = bf(((pr * back).reshape(n, -1)[:, :n] @ v[:, kv] / total).float()).double()
    return exact, rounded


def check(got, exact, rounded):
    rms = lambda e: float((e ** 2).mean().sqrt())
    a, b = rms(got.double() - exact), rms(rounded - exact)
    # a few hundred thousand roundings on either side: each root mean square is known to a few tenths of a percent
    assert a < 1.01 * b, (a, b, a / b)


@pytest.mark.parametrize("n,new", [(700, 700), (512, 100), (2000, 2000)])
@pytest.mark.parametrize("deviation", [1, 2, 4, 8])
def test_pages(n, new, deviation):
    from kubeai_b200 import ops
    heads, kv_heads, D = 4, 1, 128
    g = torch.Generator(device=DEV).manual_seed(n + deviation)
    qkv = bf(torch.randn(n, (heads + 2 * kv_heads) * D, generator=g, device=DEV))
    pages = -(-n // 16)
    order = torch.randperm(pages, generator=g, device=DEV)
    rows = torch.zeros(pages * 16, 2, kv_heads, D, dtype=torch.bfloat16, device=DEV)
    rows[:n] = qkv[:, heads * D:].reshape(n, 2, kv_heads, D)
    kv = torch.zeros(pages, 2, kv_heads, 16, D, dtype=torch.bfloat16, device=DEV)
    kv[order] = rows.reshape(pages, 16, 2, kv_heads, D).permute(0, 2, 3, 1, 4)
    q = qkv.clone()
    q[:, :heads * D] *= deviation                # a power of two: exact
    work = torch.tensor([[j, min(64, new - j), n - new + j, 0] for j in range(0, new, 64)], dtype=torch.int32, device=DEV)
    got = ops.paged_attn_prefill_tc(q[n - new:].contiguous(), kv, order.to(torch.int32)[None].contiguous(), work, heads, kv_heads)
    q64 = q[:, :heads * D].reshape(n, heads, D).double()
    exact, rounded = attention(q64, rows[:n, 0].double(), rows[:n, 1].double(), D ** -0.5, rounded_sum=False)
    check(got.reshape(new, heads, D), exact[n - new:], rounded[n - new:])


@pytest.mark.parametrize("lens", [[700], [64, 1, 513, 65]])
@pytest.mark.parametrize("deviation", [1, 3, 6, 12])
@pytest.mark.parametrize("form", ["plain", "cap", "window", "sink", "terms", "terms, cap, window, sink"])
def test_whole_prompts(lens, deviation, form):
    from kubeai_b200 import ops
    terms, cap, window, sink = "terms" in form, 5.0 * deviation if "cap" in form else 0.0, 100 if "window" in form else 0, "sink" in form
    heads, kv_heads, T = 4, 4 if terms else 2, sum(lens)
    g = torch.Generator(device=DEV).manual_seed(deviation + len(form))
    r = lambda *shape: torch.randn(*shape, generator=g, device=DEV)
    q, kv, scale = bf(r(T, heads, 128)), bf(r(T, kv_heads, 256)), deviation / math.sqrt(192 if terms else 128)
    q2, k2, v2 = (bf(r(T, heads, 64)), bf(r(T, 64)), bf(2.0 ** -9 * r(T, heads, 128))) if terms else (None, None, None)
    sinks = deviation * r(heads) if sink else None
    got = ops.prompt_attn(q, kv, lens, scale, q2=q2, k2=k2, v2=v2, window=window, softcap=cap, sink=sinks)
    parts, at = [], 0
    for n in lens:
        at, s = at + n, slice(at, at + n)
        qd, kd, vd = q[s].double(), kv[s, :, :128].double(), kv[s, :, 128:].double()
        if terms:
            qd, vd = torch.cat([qd, q2[s].double()], 2), vd + v2[s].double()
            kd = torch.cat([kd, k2[s, None].double().expand(-1, kv_heads, -1)], 2)
        parts.append(attention(qd, kd, vd, scale, rounded_sum=True, cap=cap, window=window, sink=sinks))
    check(got, torch.cat([a for a, _ in parts]), torch.cat([b for _, b in parts]))
