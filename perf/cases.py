"""The calls whose speed this framework is measured by, with their inputs, the least work each needs and its values in 64 bits.

A user of the framework feeds sequences to an engine (kubeai_b200.engine.Engine) and reads logits: whole prompts in one
step (prefill), then one token per sequence and step (decode).  The cases are such calls on the built-in Llama kernel
sequence at the layer sizes of Llama-3-8B and on registered designs at the "w2048" sizes of kubeai_b200/design_bench.py,
with few layers, each kind of layer once, and three single operations of kubeai_b200.ops at Llama-3-8B sizes.

Weights belong to a case's family and are the same for every seed; a seed makes the tokens (or the operands of an
operation).  An engine serves all states of its family, as a server's engine serves all its requests.  Routers are made
decisive the way trained ones are: every token's embedding leans towards two experts, so that rounding decides no route.

Every engine runs bf16 storage: the fp32 storage mode exists to check it and serves nothing.
"""
import json
import math
import os
import struct
import tempfile

import numpy as np
import torch

DEV = "cuda"
VOCAB = 8192
# serving limits of every engine here
MAX_SEQS, MAX_TOKENS, MAX_LEN, KV_BLOCKS = 128, 4096, 4096, 16384

# Llama-3-8B's layer
HID, QH, KVH, HD, INTER, THETA, EPS = 4096, 32, 8, 128, 14336, 500000.0, 1e-5
LLAMA_LAYERS = 2
PROJ = {"qkv": ((QH + 2 * KVH) * HD, HID), "o": (HID, QH * HD), "gate_up": (2 * INTER, HID), "down": (HID, INTER)}

# the design benchmark's size "w2048"
W, H, D, ROT, RANK, FF, EXPERTS, EFF, TOP, GROUPS, KEEP, WINDOW = 2048, 16, 128, 64, 512, 8192, 16, 2048, 2, 4, 2, 1024


def listed():
    return [
        # one user typing: a short prompt, then tokens one by one; every launch and every wait shows
        dict(name="llama chat, 1 sequence", kind="engine", family="llama", seqs=1, prompt=24, steps=16),
        # the batch of a busy replica: 128 sequences of unequal length, one token each per step
        dict(name="llama chat, 128 sequences", kind="engine", family="llama", seqs=128, prompt=2560, steps=12),
        # a burst of arriving prompts in one step
        dict(name="llama prefill, 2048 tokens", kind="engine", family="llama", seqs=5, prompt=2048, steps=0),
        # the attention of a decode step over long ragged contexts, the part that grows with the conversations
        dict(name="decode attention, 128 x 2048", kind="attention", seqs=128, ctx=2048),
        # the feed-forward's first product for a few sequences: a pass over the weights
        dict(name="gate and up, 16 tokens", kind="gate_up", tokens=16),
        # a projection of an odd-sized burst
        dict(name="down projection, 1999 tokens", kind="linear", proj="down", tokens=1999),
        # prompts through each registered design's layers: softmax attention with capped scores, matrix memory, experts
        dict(name="mulenex prefill, 4096 tokens", kind="engine", family="mulenex", seqs=8, prompt=4096, steps=0),
        # latent attention, gated linear attention, a dense and an expert feed-forward
        dict(name="nomanex prefill, 3001 tokens", kind="engine", family="nomanex", seqs=6, prompt=3001, steps=0),
        # latent attention with a query latent, two kinds of recurrence, dense feed-forwards
        dict(name="soselix prefill, 4096 tokens", kind="engine", family="soselix", seqs=3, prompt=4096, steps=0),
        # windowed attention, the gated delta rule, grouped experts
        dict(name="dabodra prefill, 4095 tokens", kind="engine", family="dabodra", seqs=8, prompt=4095, steps=0),
        # conversations on two designs: short prompts, then token by token
        dict(name="mulenex chat, 24 sequences", kind="engine", family="mulenex", seqs=24, prompt=500, steps=16),
        dict(name="soselix chat, 8 sequences", kind="engine", family="soselix", seqs=8, prompt=250, steps=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prefill", "prefill", "prefill", "chat", "chat", "chat", "attention", "gate_up", "linear"])
    if kind == "attention":
        return dict(kind="attention", seqs=rng.randint(19, 128), ctx=_log_int(rng, 48, 2048))
    if kind == "gate_up":
        return dict(kind="gate_up", tokens=_log_int(rng, 1, 128))
    if kind == "linear":
        return dict(kind="linear", proj=rng.choice(sorted(PROJ)), tokens=_log_int(rng, 129, 2048))
    family = rng.choice(["llama", "mulenex", "nomanex", "soselix", "dabodra"])
    if kind == "prefill":
        seqs = rng.randint(1, 12)
        most = 2048 if family == "llama" else 4096
        return dict(kind="engine", family=family, seqs=seqs, prompt=max(8 * seqs, _log_int(rng, 64, most)), steps=0)
    seqs = _log_int(rng, 1, 128)
    return dict(kind="engine", family=family, seqs=seqs, prompt=seqs * rng.randint(4, 24), steps=rng.randint(4, 16))


# ---------------------------------------------------------------- what a case feeds
def _lens(case):
    """Prompt lengths of the sequences: unequal, from short to long."""
    n = case["seqs"]
    return [max(1, case["prompt"] * (2 * i + 1) // (n * n)) for i in range(n)]


def _tokens(case, seed):
    g = torch.Generator().manual_seed(1000003 * (seed + 1))
    return [torch.randint(0, VOCAB, (n + case["steps"],), generator=g).numpy().astype(np.int32) for n in _lens(case)]


def _prompt_wants(case):
    """Positions of each prompt whose logits are read: the last one and, of few sequences, some evenly before it."""
    per = max(1, 32 // case["seqs"])
    return [sorted({(n * (j + 1)) // per - 1 for j in range(per) if (n * (j + 1)) // per >= 1}) for n in _lens(case)]


def _step_wants(case):
    """Sequences whose logits a decode step reads: all of a small batch, about 16 of a large one."""
    return list(range(0, case["seqs"], max(1, case["seqs"] // 16)))


def _contexts(case):
    return [max(1, case["ctx"] * (2 * i + 1) // (2 * case["seqs"])) for i in range(case["seqs"])]


# ---------------------------------------------------------------- the families' configurations and weights
def _config(family):
    moe = dict(kind="moe", expert=dict(ff=EFF), router=dict(experts=EXPERTS, top=TOP))
    if family == "mulenex":
        at = dict(heads=H, kv_heads=H // 4, dim=D, vdim=D, scale=D ** -0.5, softcap=30.0, q_temp=dict(coef=0.1, every=256), v_mix=True)
        moe["shared"] = dict(ff=EFF)
        layers = [dict(type="attention", mixer=at, mlp=moe), dict(type="mlstm", mixer=dict(heads=H, dim=D, vdim=D, gate_cap=15.0), mlp=moe)]
        return dict(architecture="Mulenex", vocab=VOCAB, width=W, norm=dict(eps=EPS), layers=layers)
    if family == "nomanex":
        la = dict(heads=H, dim=D, rot_dim=ROT, vdim=D, kv_rank=RANK, mask=dict(size=WINDOW), rot=dict(base=10000.0, dims=ROT), scale=(D + ROT) ** -0.5)
        moe["router"]["groups"] = dict(count=GROUPS, keep=KEEP)
        layers = [dict(type="latent_attention", mixer=la, mlp=dict(kind="dense", ff=FF, limit=7.0)),
                  dict(type="gla", mixer=dict(heads=H, dim=D, vdim=D, tau=16.0), mlp=moe)]
        return dict(architecture="Nomanex", vocab=VOCAB, width=W, residual_mult=0.5, norm=dict(eps=EPS),
                    embedding=dict(bigram=dict(buckets=65521, mul_prev=127, mul_cur=17)), layers=layers)
    if family == "soselix":
        la = dict(heads=H, dim=D, rot_dim=ROT, vdim=D, kv_rank=RANK, q_rank=W // 2, rot=dict(base=10000.0, dims=ROT), scale=(D + ROT) ** -0.5)
        ma = dict(heads=2 * W // 64, vdim=64, state=128, groups=8, norm_groups=8, conv=4)
        dn = dict(kind="dense", ff=FF)
        layers = [dict(type="latent_attention", mixer=la, mlp=dn), dict(type="hgrn2", mixer=dict(heads=H, dim=D, vdim=D), mlp=dn),
                  dict(type="mamba2", mixer=ma, mlp=dn)]
        return dict(architecture="Soselix", vocab=VOCAB, width=W, residual_mult=0.5, norm=dict(eps=EPS), embedding=dict(scale=1.0), layers=layers)
    if family == "dabodra":
        at = dict(heads=H, kv_heads=H // 4, dim=D, vdim=D, mask=dict(size=WINDOW), rot=dict(base=10000.0, dims=ROT), scale=D ** -0.5)
        moe["router"].update(groups=dict(count=GROUPS, keep=KEEP), scale=1.0)
        moe["shared"] = dict(ff=EFF)
        layers = [dict(type="attention", mixer=at, mlp=moe), dict(type="delta", mixer=dict(heads=H, kv_heads=H, dim=D, vdim=D, conv=4), mlp=moe)]
        return dict(architecture="Dabodra", vocab=VOCAB, width=W, norm=dict(eps=EPS), layers=layers)
    raise ValueError(family)


def _weights(family):
    """name -> bf16 tensor on the GPU, the same for every seed."""
    g = torch.Generator(device=DEV).manual_seed(sum(map(ord, family)))
    P = {}

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device=DEV)

    def put(name, t):
        P[name] = t.to(torch.bfloat16)

    def mat(name, rows, cols, gain=1.0):
        put(name, rnd(rows, cols) * (gain / math.sqrt(cols)))

    def vec(name, n, mean=0.0, dev=0.1):
        put(name, mean + dev * rnd(n))

    if family == "llama":
        put("embed", rnd(VOCAB, HID))
        for i in range(LLAMA_LAYERS):
            p = "layers.%d." % i
            for name, key in (("wqkv", "qkv"), ("wo", "o"), ("wgu", "gate_up"), ("wdown", "down")):
                mat(p + name, *PROJ[key])
            vec(p + "norm1", HID, 1.0)
            vec(p + "norm2", HID, 1.0)
        vec("final_norm", HID, 1.0)
        mat("lm_head", VOCAB, HID)
        return P
    cfg = _config(family)
    embed = rnd(VOCAB, W)
    lean = rnd(EXPERTS, W)
    lean = lean / lean.norm(dim=1, keepdim=True)             # one direction per expert, shared by the layers' routers
    if any(ly["mlp"]["kind"] == "moe" for ly in cfg["layers"]):
        first = torch.randint(0, EXPERTS, (VOCAB,), generator=g, device=DEV)
        second = (first + 1 + torch.randint(0, EXPERTS - 1, (VOCAB,), generator=g, device=DEV)) % EXPERTS
        embed = embed + 14.0 * lean[first] + 11.0 * lean[second]
    put("embed", embed)
    mat("head", VOCAB, W)
    if family == "mulenex":
        vec("final.norm", W)
        for i, ly in enumerate(cfg["layers"]):
            p = "l%d." % i
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                vec(p + n, W)
            if ly["type"] == "attention":
                mat(p + "mix.q", H * D, W)
                mat(p + "mix.k", H // 4 * D, W)
                mat(p + "mix.v", H // 4 * D, W)
                mat(p + "mix.g", H, W)
                vec(p + "mix.q.norm", D, 1.0)
                vec(p + "mix.k.norm", D, 1.0)
                put(p + "mix.vmix", torch.tensor(0.5, device=DEV))
            else:
                for n in "qkvg":
                    mat(p + "mix." + n, H * D, W)
                # queries lean towards their own token's key: the memory's answer has a sign that rounding does not turn
                put(p + "mix.q", 0.8 * P[p + "mix.k"].float() + 0.6 * P[p + "mix.q"].float())
                vec(p + "mix.norm", H * D, 1.0)
                for n, mean in (("i", 0.0), ("f", 3.0)):
                    mat(p + "mix." + n, H, W)
                    vec(p + "mix.%s.b" % n, H, mean, 0.5)
            mat(p + "mix.o", W, H * D)
            put(p + "mlp.router", 0.3 * lean)
            vec(p + "mlp.router.b", EXPERTS, 0.0, 0.05)
            for n in ["e%d" % e for e in range(EXPERTS)] + ["shared"]:
                mat(p + "mlp.%s.gate" % n, EFF, W, 1.5)
                mat(p + "mlp.%s.up" % n, EFF, W, 1.5)
                mat(p + "mlp.%s.down" % n, W, EFF)
            mat(p + "mlp.shared.sg", 1, W)
    elif family == "nomanex":
        def dyt(name):
            vec(name, W, 1.0)
            vec(name + ".b", W)
            put(name + ".alpha", torch.tensor(0.75, device=DEV))

        put("bigram", 0.3 * rnd(65522, W))
        dyt("final.norm")
        for i, ly in enumerate(cfg["layers"]):
            p = "l%d." % i
            dyt(p + "norm1")
            if ly["type"] == "gla":
                for n in "qkvg":
                    mat(p + "mix." + n, H * D, W, 1.5)
                mat(p + "mix.a1", 16, W)
                mat(p + "mix.a2", H * D, 16)
                vec(p + "mix.a2.b", H * D, 2.0, 1.0)
                vec(p + "mix.norm", D, 1.0)
            else:
                mat(p + "mix.q", H * (D + ROT), W, 1.5)
                mat(p + "mix.dkv", RANK + ROT, W, 1.5)
                vec(p + "mix.dkv.norm", RANK, 1.0)
                mat(p + "mix.uk", H * D, RANK)
                mat(p + "mix.uv", H * D, RANK)
                mat(p + "mix.g", H * D, W)
            mat(p + "mix.o", W, H * D, 1.5)
            if ly["mlp"]["kind"] == "dense":
                mat(p + "mlp.gate", FF, W, 1.5)
                mat(p + "mlp.up", FF, W, 1.5)
                mat(p + "mlp.down", W, FF)
            else:
                put(p + "mlp.router", 0.7 * lean)
                for e in range(EXPERTS):
                    mat(p + "mlp.e%d.up" % e, EFF, W, 1.5)
                    mat(p + "mlp.e%d.down" % e, W, EFF)
    elif family == "soselix":
        put("final.norm", torch.tensor(1.1, device=DEV))
        for i, ly in enumerate(cfg["layers"]):
            p, mx = "l%d." % i, ly["mixer"]
            put(p + "norm1", torch.tensor(0.9, device=DEV))
            put(p + "norm2", torch.tensor(1.1, device=DEV))
            if ly["type"] == "latent_attention":
                mat(p + "mix.dq", W // 2, W)
                vec(p + "mix.dq.norm", W // 2, 1.0)
                mat(p + "mix.uq", H * (D + ROT), W // 2, 1.5)
                mat(p + "mix.dkv", RANK + ROT, W)
                vec(p + "mix.dkv.norm", RANK, 1.0)
                mat(p + "mix.uk", H * D, RANK)
                mat(p + "mix.uv", H * D, RANK)
                vec(p + "mix.sink", H, 0.5, 1.0)
                mat(p + "mix.g", H, W)
                out = H * D
            elif ly["type"] == "hgrn2":
                for n in "qfv":
                    mat(p + "mix." + n, H * D, W, 1.5)
                vec(p + "mix.f.b", H * D, 1.0, 1.0)
                put(p + "mix.lower", 0.9 * torch.rand(H * D, generator=g, device=DEV))
                vec(p + "mix.norm", D, 1.0)
                out = H * D
            else:
                Hm, P_, N, G = mx["heads"], mx["vdim"], mx["state"], mx["groups"]
                ch = Hm * P_ + 2 * G * N
                mat(p + "mix.in", Hm * P_ + ch + Hm, W, 1.5)
                put(p + "mix.conv", 0.6 * rnd(ch, mx["conv"]))
                vec(p + "mix.conv.b", ch, 0.0, 0.2)
                vec(p + "mix.dt_bias", Hm, -2.0, 1.0)
                put(p + "mix.A_log", torch.log(0.05 + 3.95 * torch.rand(Hm, generator=g, device=DEV)))
                vec(p + "mix.D", Hm, 1.0, 0.2)
                vec(p + "mix.norm", Hm * P_, 1.0)
                out = Hm * P_
            mat(p + "mix.o", W, out, 1.5)
            mat(p + "mlp.up", FF, W, 1.5)
            vec(p + "mlp.up.b", FF, 0.0, 0.2)
            mat(p + "mlp.down", W, FF)
            vec(p + "mlp.down.b", W, 0.0, 0.2)
            vec(p + "mlp.act", 2, 0.0, 0.5)
    elif family == "dabodra":
        vec("embed.norm", W)
        vec("final.norm", W)
        for i, ly in enumerate(cfg["layers"]):
            p = "l%d." % i
            vec(p + "norm1", W)
            vec(p + "norm2", W)
            if ly["type"] == "attention":
                mat(p + "mix.q", H * D, W)
                mat(p + "mix.k", H // 4 * D, W)
                vec(p + "mix.q.norm", H * D, 1.0)
                vec(p + "mix.k.norm", H // 4 * D, 1.0)
                vec(p + "mix.sink", H, 0.5, 1.0)
            else:
                for n in "qkv":
                    mat(p + "mix." + n, H * D, W, 1.5)
                    put(p + "mix.%s.conv" % n, 0.6 * rnd(H * D, 4))
                mat(p + "mix.b", H, W)
                mat(p + "mix.a", H, W)
                put(p + "mix.A_log", -2.0 + 3.0 * torch.rand(H, generator=g, device=DEV))
                vec(p + "mix.dt_bias", H, -1.5, 1.0)
                vec(p + "mix.norm", D, 1.0)
                mat(p + "mix.g", H * D, W, 1.5)
            mat(p + "mix.o", W, H * D)
            put(p + "mlp.router", 0.25 * lean)
            vec(p + "mlp.correction", EXPERTS, 0.0, 0.02)
            for n in ["e%d" % e for e in range(EXPERTS)] + ["shared"]:
                mat(p + "mlp.%s.gate" % n, EFF, W, 1.5)
                mat(p + "mlp.%s.up" % n, EFF, W, 1.5)
                mat(p + "mlp.%s.down" % n, W, EFF)
    return P


def _bits(t):
    return t.contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


def _write_model_dir(d, cfg, P):
    """config.json and model.safetensors: an 8-byte header length, the JSON header, the tensors one after the other."""
    with open(os.path.join(d, "config.json"), "w") as f:
        json.dump(cfg, f)
    header, at = {}, 0
    for name, t in P.items():
        header[name] = dict(dtype="BF16", shape=list(t.shape), data_offsets=[at, at + 2 * t.numel()])
        at += 2 * t.numel()
    hj = json.dumps(header).encode()
    with open(os.path.join(d, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(hj)) + hj)
        for t in P.values():
            f.write(memoryview(_bits(t).reshape(-1)))


_live = {}   # the engine of the family in use: a program serves one model


def _engine(family):
    if family not in _live:
        from kubeai_b200.engine import Engine, default_config
        for e in _live.values():
            e.close()
        _live.clear()
        lim = dict(max_model_len=MAX_LEN, max_num_seqs=MAX_SEQS, max_batched_tokens=MAX_TOKENS, num_kv_blocks=KV_BLOCKS, enable_prefix_caching=0,
                   manual_step=1, eos_token_id=-1)
        P = _weights(family)
        if family == "llama":
            e = Engine(default_config(num_layers=LLAMA_LAYERS, hidden=HID, q_heads=QH, kv_heads=KVH, intermediate=INTER, vocab=VOCAB,
                                      rms_eps=EPS, rope_theta=THETA, **lim))
            for name, t in P.items():
                e.tensor_write(name, _bits(t))
        else:
            shm = "/dev/shm" if os.path.isdir("/dev/shm") else None
            with tempfile.TemporaryDirectory(dir=shm) as d:
                _write_model_dir(d, _config(family), P)
                e = Engine(default_config(**lim), d, dtype="bfloat16")
        _live[family] = e
    return _live[family]


# ---------------------------------------------------------------- inputs and passes
def _attention_inputs(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    n, ctxs = case["seqs"], _contexts(case)
    pages = [(c + 15) // 16 for c in ctxs]
    total = sum(pages)
    order = torch.randperm(total, generator=g, device=DEV).to(torch.int32)       # a pool in use is not in order
    tables = torch.zeros(n, max(pages), dtype=torch.int32, device=DEV)
    at = 0
    for i, m in enumerate(pages):
        tables[i, :m] = order[at:at + m]
        at += m
    qkv = torch.randn(n, (QH + 2 * KVH) * HD, generator=g, device=DEV).to(torch.bfloat16)
    kv = torch.randn(total, 2, KVH, 16, HD, generator=g, device=DEV, dtype=torch.bfloat16)
    work = torch.tensor([[i, 1, c - 1, i] for i, c in enumerate(ctxs)], dtype=torch.int32, device=DEV)
    return dict(qkv=qkv, kv=kv, tables=tables, work=work)


def _linear_inputs(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    n, k = PROJ["gate_up" if case["kind"] == "gate_up" else case["proj"]]
    x = torch.randn(case["tokens"], k, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).to(torch.bfloat16)
    return dict(x=x, w=w)


def prepare(case, seed):
    if case["kind"] == "attention":
        return dict(case=case, **_attention_inputs(case, seed))
    if case["kind"] in ("gate_up", "linear"):
        return dict(case=case, **_linear_inputs(case, seed))
    toks, lens = _tokens(case, seed), _lens(case)
    prompt = [(t[:n], np.asarray(w, dtype=np.int32)) for t, n, w in zip(toks, lens, _prompt_wants(case))]
    read = set(_step_wants(case))
    none, this = np.zeros(0, dtype=np.int32), np.zeros(1, dtype=np.int32)
    steps = [[(t[n + s:n + s + 1], this if i in read else none) for i, (t, n) in enumerate(zip(toks, lens))] for s in range(case["steps"])]
    return dict(case=case, engine=_engine(case["family"]), prompt=prompt, steps=steps)


def run(state):
    kind = state["case"]["kind"]
    if kind == "engine":
        e = state["engine"]
        ids = [e.feed_open() for _ in state["prompt"]]
        out = [e.feed_step([(r, t, w) for r, (t, w) in zip(ids, state["prompt"])])]
        for entries in state["steps"]:
            out.append(e.feed_step([(r, t, w) for r, (t, w) in zip(ids, entries)]))
        for r in ids:
            e.feed_close(r)
        return out
    from kubeai_b200 import ops
    if kind == "attention":
        return ops.paged_attn(state["qkv"], state["kv"], state["tables"], state["work"], QH, KVH, decode=True)
    if kind == "gate_up":
        return ops.gemm3(state["x"], state["w"], epi=ops.EPI_SILU)[0]
    return ops.gemm(state["x"], state["w"])


# ---------------------------------------------------------------- the least work of a pass
def _family_work(family):
    """(weights every token passes, weights of one routed expert summed over the expert layers, score and value products
    per query and key pair, cache values a token leaves, state values of a sequence, recurrence products per token)."""
    if family == "llama":
        return LLAMA_LAYERS * sum(a * b for a, b in PROJ.values()), 0, LLAMA_LAYERS * QH * 2 * HD, LLAMA_LAYERS * 2 * KVH * HD, 0, 0
    if family == "mulenex":
        dense = W * (H * D + 2 * (H // 4) * D + H) + H * D * W + W * (4 * H * D + 2 * H) + H * D * W + 2 * (3 * W * EFF + W * EXPERTS)
        return dense, 2 * 3 * W * EFF, H * 2 * D, 2 * (H // 4) * D, H * D * D, 3 * H * D * D
    if family == "nomanex":
        dense = W * (H * (D + ROT) + RANK + ROT + H * D) + 2 * H * D * RANK + H * D * W + 3 * W * FF
        dense += W * 4 * H * D + 16 * (W + H * D) + H * D * W + W * EXPERTS
        return dense, 2 * W * EFF, H * (2 * D + ROT), RANK + ROT, H * D * D, 3 * H * D * D
    if family == "soselix":
        Hm, P_, N, G = 2 * W // 64, 64, 128, 8
        dense = W * (W // 2 + RANK + ROT + H) + W // 2 * H * (D + ROT) + 2 * H * D * RANK + H * D * W
        dense += W * 3 * H * D + H * D * W + W * (2 * Hm * P_ + 2 * G * N + Hm) + Hm * P_ * W + 3 * 2 * W * FF
        return dense, 0, H * (2 * D + ROT), RANK + ROT, H * D * D + Hm * N * P_, 3 * (H * D * D + Hm * N * P_)
    dense = W * (H * D + (H // 4) * D) + H * D * W + W * (4 * H * D + 2 * H) + H * D * W + 2 * (3 * W * EFF + W * EXPERTS)
    return dense, 2 * 3 * W * EFF, H * 2 * D, 2 * (H // 4) * D, H * D * D, 4 * H * D * D


def _pairs(family, n):
    """Query and key pairs of a causal sequence of n tokens, inside the family's window."""
    win = WINDOW if family in ("nomanex", "dabodra") else n
    return sum(min(p + 1, win) for p in range(n))


def work(case):
    if case["kind"] == "attention":
        keys = sum(_contexts(case))
        return dict(bytes=keys * 2 * KVH * HD * 2 + case["seqs"] * 2 * QH * HD * 2, flops=4 * keys * QH * HD)
    if case["kind"] in ("gate_up", "linear"):
        n, k = PROJ["gate_up" if case["kind"] == "gate_up" else case["proj"]]
        t = case["tokens"]
        return dict(bytes=2 * (n * k + t * k + t * (n // 2 if case["kind"] == "gate_up" else n)), flops=2 * n * k * t)
    f, lens, steps = case["family"], _lens(case), case["steps"]
    dense, expert, per_pair, cached, state, recur = _family_work(f)
    read = sum(len(w) for w in _prompt_wants(case)) + steps * len(_step_wants(case))
    tokens = sum(lens) + steps * len(lens)
    flops = 2 * tokens * (dense + TOP * expert) + 2 * read * VOCAB * (HID if f == "llama" else W)
    flops += 2 * per_pair * sum(_pairs(f, n + steps) for n in lens) + 2 * recur * tokens
    size = 0
    for s in range(steps + 1):
        t = sum(lens) if s == 0 else len(lens)
        hit = EXPERTS * (1 - (1 - 1 / EXPERTS) ** (TOP * t))           # experts that some token is routed to
        rows = sum(len(w) for w in _prompt_wants(case)) if s == 0 else len(_step_wants(case))
        size += 2 * (dense + hit * expert) + (2 * VOCAB * (HID if f == "llama" else W) if rows else 0) + 4 * rows * VOCAB
        size += len(lens) * state * 4 * (1 if s == 0 else 2)
        size += 2 * cached * (sum(lens) if s == 0 else sum(min(n + s, WINDOW) if f in ("nomanex", "dabodra") else n + s for n in lens))
    return dict(bytes=size, flops=flops)


def tolerance(case):
    # one product or one softmax in bf16 with 32-bit sums: half an ulp of bf16 (2^-9) at worst, another order of the sums
    # moves few elements by one ulp
    if case["kind"] != "engine":
        return dict(rel=4e-3, max=0.05)
    # several layers in bf16: another order of sums moves some roundings in every layer, and these travel on
    return dict(rel=2e-2, max=0.3)


# ---------------------------------------------------------------- the same values in 64 bits
def _unit(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, dims, base, pairs):
    """Rotate the first `dims` entries of x [n, L, heads, d] by the position; entry i pairs with i + dims / 2, or 2i with 2i + 1."""
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / dims)
    ang = torch.arange(x.shape[1], device=x.device, dtype=torch.float64)[:, None] * f
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    out = x.clone()
    ia, ib = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, half), slice(half, dims))
    a, b = x[..., ia], x[..., ib]
    out[..., ia] = a * c - b * s
    out[..., ib] = b * c + a * s
    return out


def _attend(q, k, v, scale, window=None, cap=None, sink=None):
    """Causal softmax attention, q [n, L, heads, d], k and v [n, L, key heads, d]."""
    n, L, heads, _ = q.shape
    G = k.shape[2]
    out = torch.empty(n, L, heads, v.shape[-1], dtype=q.dtype, device=q.device)
    i = torch.arange(L, device=q.device)
    hide = i[None, :] > i[:, None]
    if window:
        hide = hide | (i[:, None] - i[None, :] >= window)
    for s in range(n):
        for h in range(heads):
            g = h // (heads // G)
            z = (q[s, :, h] @ k[s, :, g].T) * scale
            if cap:
                z = cap * torch.tanh(z / cap)
            z = z.masked_fill(hide, -math.inf)
            if sink is not None:
                z = torch.cat([z, sink[h].expand(L, 1)], 1)
            w = torch.softmax(z, 1)[:, :L]
            out[s, :, h] = w @ v[s, :, g]
    return out


def _scan(decay, k, v, q):
    """S <- decay S + k v^T, o = S^T q; decay [n, L, heads, d or 1], k and q [n, L, heads, d], v [n, L, heads, dv]."""
    n, L, heads, d = k.shape
    S = torch.zeros(n, heads, d, v.shape[-1], dtype=k.dtype, device=k.device)
    o = torch.empty(n, L, heads, v.shape[-1], dtype=k.dtype, device=k.device)
    for t in range(L):
        S = S * decay[:, t, :, :, None] + k[:, t, :, :, None] * v[:, t, :, None, :]
        o[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
    return o


def _conv(u, w, b=0.0):
    taps = w.shape[1]
    pad = torch.nn.functional.pad(u, (0, 0, taps - 1, 0))
    return sum(pad[:, j:j + u.shape[1]] * w[:, j] for j in range(taps)) + b


def _gated(p, pre, x):
    return (_silu(x @ p(pre + "gate").T) * (x @ p(pre + "up").T)) @ p(pre + "down").T


def _experts(x, pick, weight, one):
    """Sum over the chosen experts of weight times one(expert, rows)."""
    flat, out = x.reshape(-1, x.shape[-1]), torch.zeros_like(x).reshape(-1, x.shape[-1])
    pick, weight = pick.reshape(-1, pick.shape[-1]), weight.reshape(-1, pick.shape[-1])
    for e in range(EXPERTS):
        rows, col = torch.nonzero(pick == e, as_tuple=True)
        if len(rows):
            out.index_add_(0, rows, weight[rows, col][:, None] * one(e, flat[rows]))
    return out.reshape(x.shape)


def _open_groups(score, rank):
    """The scores with those outside the kept groups at -inf; rank: a group's rank from its members' scores."""
    parts = score.reshape(*score.shape[:-1], GROUPS, EXPERTS // GROUPS)
    best = rank(parts).topk(KEEP, -1).indices
    keep = torch.zeros(parts.shape[:-1], dtype=torch.bool, device=score.device).scatter_(-1, best, True)
    return parts.masked_fill(~keep[..., None], -math.inf).reshape(score.shape)


def _forward64(family, ids):
    """Final normed residual [n, L, width] of the padded sequences ids [n, L], and the head."""
    P = _weights(family)
    dims = ids.shape

    def p(name):
        return P[name].double()

    def heads(x, h):
        return x.reshape(*dims, h, -1)

    if family == "llama":
        x = p("embed")[ids]
        for i in range(LLAMA_LAYERS):
            a = "layers.%d." % i
            y = (_unit(x) * p(a + "norm1")) @ p(a + "wqkv").T
            q, k, v = (heads(t, h) for t, h in zip(y.split([QH * HD, KVH * HD, KVH * HD], -1), (QH, KVH, KVH)))
            o = _attend(_rotate(q, HD, THETA, False), _rotate(k, HD, THETA, False), v, HD ** -0.5)
            x = x + o.reshape(*dims, -1) @ p(a + "wo").T
            gu = (_unit(x) * p(a + "norm2")) @ p(a + "wgu").T
            x = x + (_silu(gu[..., :INTER]) * gu[..., INTER:]) @ p(a + "wdown").T
        return _unit(x) * p("final_norm"), p("lm_head")
    layers = _config(family)["layers"]
    if family == "mulenex":
        pos = torch.arange(dims[1], device=DEV, dtype=torch.float64)[:, None]
        c = torch.arange(W, device=DEV)
        ang = pos * 10000.0 ** (-2.0 * torch.div(c, 2, rounding_mode="floor").double() / W)
        x = p("embed")[ids] + torch.where(c % 2 == 0, torch.sin(ang), torch.cos(ang))
        for i, ly in enumerate(layers):
            a = "l%d." % i
            h = _unit(x) * (1 + p(a + "norm1"))
            m = a + "mix."
            if ly["type"] == "attention":
                temp = 1 + 0.1 * torch.log(torch.floor((pos + 1) / 256) + 1)
                q = _unit(heads(h @ p(m + "q").T, H)) * p(m + "q.norm") * temp[:, :, None]
                k = _unit(heads(h @ p(m + "k").T, H // 4)) * p(m + "k.norm")
                o = _attend(q, k, heads(h @ p(m + "v").T, H // 4), D ** -0.5, cap=30.0)
                o = o * torch.sigmoid(h @ p(m + "g").T)[..., None]
            else:
                q, k, v = (heads(h @ p(m + n).T, H) for n in "qkv")
                li, lf = (15.0 * torch.tanh((h @ p(m + n).T + p(m + n + ".b")) / 15.0) for n in "if")
                lf = torch.nn.functional.logsigmoid(lf)
                top, keep, take = torch.zeros(dims[0], H, dtype=x.dtype, device=DEV), torch.empty_like(lf), torch.empty_like(lf)
                tops = torch.empty_like(lf)
                for t in range(dims[1]):
                    new = torch.maximum(lf[:, t] + top, li[:, t])
                    keep[:, t], take[:, t], tops[:, t] = torch.exp(lf[:, t] + top - new), torch.exp(li[:, t] - new), new
                    top = new
                one = torch.ones(*dims, H, 1, dtype=x.dtype, device=DEV)
                o = _scan(keep[..., None], k * take[..., None], torch.cat([v, one], -1), q * D ** -0.5)
                o = o[..., :D] / (torch.maximum(o[..., D:].abs(), torch.exp(-tops)[..., None]) + 1e-6)
                o = (_unit(o).reshape(*dims, -1) * p(m + "norm") * torch.sigmoid(h @ p(m + "g").T)).reshape(o.shape)
            x = x + _unit(o.reshape(*dims, -1) @ p(m + "o").T) * (1 + p(a + "norm1b"))
            h, m = _unit(x) * (1 + p(a + "norm2")), a + "mlp."
            z, pick = (h @ p(m + "router").T + p(m + "router.b")).topk(TOP, -1)
            y = _experts(h, pick, torch.softmax(z, -1), lambda e, r: _gated(p, m + "e%d." % e, r))
            y = y + torch.sigmoid(h @ p(m + "shared.sg").T) * _gated(p, m + "shared.", h)
            x = x + _unit(y) * (1 + p(a + "norm2b"))
        return _unit(x) * (1 + p("final.norm")), p("head")
    if family == "nomanex":
        def dyt(name, x):
            return torch.tanh(p(name + ".alpha") * x) * p(name) + p(name + ".b")

        row = torch.full_like(ids, 65521)
        row[:, 1:] = (ids[:, :-1] * 127 + ids[:, 1:] * 17) % 65521
        x = P["embed"][ids].double() + P["bigram"][row].double()
        for i, ly in enumerate(layers):
            a = "l%d." % i
            h, m = dyt(a + "norm1", x), a + "mix."
            if ly["type"] == "gla":
                q, k, v = (heads(h @ p(m + n).T, H) for n in "qkv")
                dec = torch.sigmoid((h @ p(m + "a1").T) @ p(m + "a2").T + p(m + "a2.b")) ** (1 / 16.0)
                o = _unit(_scan(heads(dec, H), k, v, q * D ** -0.5)) * p(m + "norm")
                y = o.reshape(*dims, -1) * _silu(h @ p(m + "g").T)
            else:
                y = _latent64(p, m, heads(h @ p(m + "q").T, H), h, WINDOW, None, True).reshape(*dims, -1) * torch.sigmoid(h @ p(m + "g").T)
            y = y @ p(m + "o").T
            m = a + "mlp."
            if ly["mlp"]["kind"] == "dense":
                gt = (h @ p(m + "gate").T).clamp(max=7.0)
                y = y + (gt * torch.sigmoid(1.702 * gt) * ((h @ p(m + "up").T).clamp(-7.0, 7.0) + 1)) @ p(m + "down").T
            else:
                s = torch.softmax(h @ p(m + "router").T, -1)
                wt, pick = _open_groups(s, lambda z: z.amax(-1)).topk(TOP, -1)
                y = y + _experts(h, pick, wt, lambda e, r: (r @ p(m + "e%d.up" % e).T).clamp(min=0).square() @ p(m + "e%d.down" % e).T)
            x = x + 0.5 * y
        return dyt("final.norm", x), p("head")
    if family == "soselix":
        x = p("embed")[ids]
        for i, ly in enumerate(layers):
            a, mx = "l%d." % i, ly["mixer"]
            h, m = _unit(x) * p(a + "norm1"), a + "mix."
            if ly["type"] == "latent_attention":
                cq = _unit(h @ p(m + "dq").T) * p(m + "dq.norm")
                y = _latent64(p, m, heads(cq @ p(m + "uq").T, H), h, None, p(m + "sink"), False) * torch.sigmoid(h @ p(m + "g").T)[..., None]
            elif ly["type"] == "hgrn2":
                z, low = h @ p(m + "f").T + p(m + "f.b"), p(m + "lower")
                f, w = low + (1 - low) * torch.sigmoid(z), (1 - low) * torch.sigmoid(-z)
                y = _unit(_scan(heads(f, H), heads(w, H), heads(h @ p(m + "v").T, H), _silu(heads(h @ p(m + "q").T, H)))) * p(m + "norm")
            else:
                Hm, Pv, N, G = mx["heads"], mx["vdim"], mx["state"], mx["groups"]
                z, xbc, dt = (h @ p(m + "in").T).split([Hm * Pv, Hm * Pv + 2 * G * N, Hm], -1)
                xs, B, C = _silu(_conv(xbc, p(m + "conv"), p(m + "conv.b"))).split([Hm * Pv, G * N, G * N], -1)
                xs, B, C = heads(xs, Hm), heads(B, G).repeat_interleave(Hm // G, 2), heads(C, G).repeat_interleave(Hm // G, 2)
                d = torch.nn.functional.softplus(dt + p(m + "dt_bias"), threshold=50.0)[..., None]
                y = _scan(torch.exp(-torch.exp(p(m + "A_log"))[:, None] * d), B * d, xs, C) + p(m + "D")[:, None] * xs
                y = _unit(heads(y.reshape(*dims, -1) * _silu(z), 8)).reshape(*dims, -1) * p(m + "norm")
            x = x + 0.5 * (y.reshape(*dims, -1) @ p(m + "o").T)
            h, m = _unit(x) * p(a + "norm2"), a + "mlp."
            z, act = h @ p(m + "up").T + p(m + "up.b"), torch.nn.functional.softplus(p(m + "act"))
            neg = z.clamp(max=0)
            z = torch.where(z > 0, act[0] * z * z, (0.5 + act[1]) * (torch.expm1(neg) - neg)) + 0.5 * z
            x = x + 0.5 * (z @ p(m + "down").T + p(m + "down.b"))
        return _unit(x) * p("final.norm"), p("head")
    x = _unit(p("embed")[ids]) * (1 + p("embed.norm"))
    for i, ly in enumerate(layers):
        a, m = "l%d." % i, "l%d.mix." % i
        if ly["type"] == "attention":
            k = x @ p(m + "k").T
            q = _rotate(heads(_unit(x @ p(m + "q").T) * p(m + "q.norm"), H), ROT, 10000.0, True)
            kn = _rotate(heads(_unit(k) * p(m + "k.norm"), H // 4), ROT, 10000.0, True)
            y = _attend(q, kn, heads(k, H // 4), D ** -0.5, window=WINDOW, sink=p(m + "sink"))
        else:
            q, k, v = (heads(_silu(_conv(x @ p(m + n).T, p(m + n + ".conv"))), H) for n in "qkv")
            q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            beta = torch.sigmoid(x @ p(m + "b").T)
            g = torch.exp(-torch.exp(p(m + "A_log")) * torch.nn.functional.softplus(x @ p(m + "a").T + p(m + "dt_bias"), threshold=50.0))
            S = torch.zeros(dims[0], H, D, D, dtype=x.dtype, device=DEV)
            o = torch.empty_like(v)
            for t in range(dims[1]):
                S = S * g[:, t, :, None, None]
                u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ S)[:, :, 0])
                S = S + k[:, t, :, :, None] * u[:, :, None, :]
                o[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0] * D ** -0.5
            y = _unit(o) * p(m + "norm") * _silu(heads(x @ p(m + "g").T, H))
        x = x + _unit(y.reshape(*dims, -1) @ p(m + "o").T) * (1 + p(a + "norm1"))
        m = a + "mlp."
        s = torch.sigmoid(x @ p(m + "router").T)
        pick = _open_groups(s + p(m + "correction"), lambda z: z.topk(2, -1).values.sum(-1)).topk(TOP, -1).indices
        wt = s.gather(-1, pick)
        y = _experts(x, pick, wt / (wt.sum(-1, keepdim=True) + 1e-20), lambda e, r: _gated(p, m + "e%d." % e, r)) + _gated(p, m + "shared.", x)
        x = x + _unit(y) * (1 + p(a + "norm2"))
    return _unit(x) * (1 + p("final.norm")), p("head")


def _latent64(p, m, q, h, window, sink, pairs):
    """Attention whose keys and values are rebuilt from a normed latent, and one rotated key part for all heads."""
    d = h @ p(m + "dkv").T
    c = _unit(d[..., :RANK]) * p(m + "dkv.norm")
    kr = _rotate(d[..., None, RANK:], ROT, 10000.0, pairs).expand(*h.shape[:2], H, ROT)
    k = torch.cat([(c @ p(m + "uk").T).reshape(*h.shape[:2], H, D), kr], -1)
    q = torch.cat([q[..., :D], _rotate(q[..., D:].contiguous(), ROT, 10000.0, pairs)], -1)
    return _attend(q, k, (c @ p(m + "uv").T).reshape(*h.shape[:2], H, D), (D + ROT) ** -0.5, window=window, sink=sink)


def exact(case, seed):
    if case["kind"] == "attention":
        s = _attention_inputs(case, seed)
        out = torch.empty(case["seqs"], QH * HD, dtype=torch.float64, device=DEV)
        for i, c in enumerate(_contexts(case)):
            rows = s["kv"][s["tables"][i, :(c + 15) // 16].long()].double()                  # [pages, 2, kv heads, 16, 128]
            k, v = (rows[:, j].transpose(0, 1).reshape(KVH, -1, HD)[:, :c] for j in (0, 1))
            q = s["qkv"][i, :QH * HD].double().reshape(KVH, QH // KVH, HD)
            out[i] = (torch.softmax(q @ k.transpose(1, 2) * HD ** -0.5, -1) @ v).reshape(-1)
        return out
    if case["kind"] in ("gate_up", "linear"):
        s = _linear_inputs(case, seed)
        y = s["x"].double() @ s["w"].double().T
        if case["kind"] == "linear":
            return y
        y = y.reshape(case["tokens"], -1, 2, 64)       # 64 gate rows, their 64 up rows, the next 64 gate rows, ...
        return (_silu(y[:, :, 0]) * y[:, :, 1]).reshape(case["tokens"], -1)
    toks, lens = _tokens(case, seed), _lens(case)
    ids = torch.zeros(len(toks), max(map(len, toks)), dtype=torch.long, device=DEV)
    for i, t in enumerate(toks):
        ids[i, :len(t)] = torch.from_numpy(t.astype(np.int64)).to(DEV)
    x, head = _forward64(case["family"], ids)

    def rows(at):
        return torch.stack([x[i, j] for i, j in at]) @ head.T

    out = [rows([(i, j) for i, w in enumerate(_prompt_wants(case)) for j in w])]
    return out + [rows([(i, lens[i] + s) for i in _step_wants(case)]) for s in range(case["steps"])]
