"""Single products that are under way on several streams at once: where K is cut, the parts of a tile meet in a workspace, and each stream has its own."""
import ctypes as C
import functools

import pytest
import torch

pytestmark = pytest.mark.gpu


def pairs():
    return torch.cuda.get_device_properties(0).multi_processor_count // 2


def rule(number, T, N, K):
    from kubeai_b200._lib import lib
    return lib().b200_rule_query(number, (C.c_int32 * 5)(T, N, K, pairs(), 1), 5)


def parts(T, N, K):
    return rule(11, T, N, K)


def call(kind, T, N, K, seed):
    from kubeai_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).to(torch.bfloat16)
    return (lambda: ops.gemm(x, w)) if kind == "gemm" else (lambda: ops.gemm3(x, w, epi=ops.EPI_SILU)[0])


@functools.cache
def two_streams():
    return torch.cuda.Stream(), torch.cuda.Stream()


@pytest.mark.parametrize("a,b", [
    (("silu", 64, 2048, 4096), ("silu", 64, 4096, 4096)), (("silu", 64, 2048, 4096), ("gemm", 64, 2048, 8192)), (("gemm", 512, 256, 4096), ("gemm", 100, 512, 4096)),
    (("silu", 64, 1024, 8192), ("gemm", 1000, 256, 4096))])
def test_two_streams(a, b):
    assert parts(*a[1:]) > 1 and parts(*b[1:]) > 1
    calls = [call(*a, seed=1), call(*b, seed=2)]
    alone = [f() for f in calls]
    torch.cuda.synchronize()
    streams, outs = two_streams(), [[], []]
    for _ in range(300):
        for i in (0, 1):
            with torch.cuda.stream(streams[i]):
                outs[i].append(calls[i]())
    torch.cuda.synchronize()
    for i in (0, 1):
        assert all(torch.equal(o, alone[i]) for o in outs[i])


@pytest.mark.parametrize("kind,T,N,K", [("gemm", 64, 1024, 8192), ("silu", 64, 2048, 4096)])
@pytest.mark.parametrize("warm", [False, True])
def test_captured(kind, T, N, K, warm):
    """A stream that is being captured gets no workspace: K cut over the one of all calls, or gemm3's clusters.  The sums' order differs from the eager call's."""
    assert parts(T, N, K) > 1
    f = call(kind, T, N, K, seed=5)
    want = f()
    g, s = torch.cuda.CUDAGraph(), two_streams()[0] if warm else torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        out = f()
    for _ in range(3):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert ((out.double() - want.double()).norm() / want.double().norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("T,N,K,kind", [(64, 28672, 4096, "tiles"), (33, 19456, 4096, "stream-K"), (33, 19456, 2048, "tiles"), (64, 2048, 4096, "tiles"), (112, 1024, 512, "tiles"), (113, 1024, 512, "gemm3")])
def test_schedule_that_is_reported(T, N, K, kind):
    from kubeai_b200 import ops
    x, w = torch.randn(T, K, device="cuda").to(torch.bfloat16), (torch.randn(N, K, device="cuda") / K ** 0.5).to(torch.bfloat16)
    got, (each, streamk, ctas) = ops.gemm3(x, w, epi=ops.EPI_SILU)
    if kind == "tiles":
        assert (each, streamk, ctas) == (1, 0, 2 * min(pairs(), N // 256 * -(-T // rule(10, T, N, K)) * parts(T, N, K)))
    else:
        assert streamk == (kind == "stream-K") and (streamk or ctas == N // 256 * 2 * each)
    g, u = (x.double() @ w.double().T).reshape(T, N // 128, 2, 64).transpose(1, 2).reshape(T, 2, N // 2).unbind(1)
    want = g * torch.sigmoid(g) * u
    # three roundings to bf16 and those of the two sums ahead of the unit
    assert ((got.double() - want).norm() / want.norm()).item() < 5 * 2.0 ** -9


def test_more_streams_than_have_a_workspace():
    """The 33rd stream and all behind it leave K whole: sums in another order, each call the same bits every time."""
    f = [call("gemm", 64, 512, 8192, seed=i) for i in range(45)]
    assert parts(64, 512, 8192) > 1
    base = [g() for g in f]
    streams = [torch.cuda.Stream(priority=-(i % 2)) for i in range(len(f))]
    assert len({s.cuda_stream for s in streams}) > 33
    outs = []
    for _ in range(20):
        for g, s in zip(f, streams):
            with torch.cuda.stream(s):
                outs.append(g())
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        k = i % len(f)
        assert torch.equal(o, outs[k])
        # fp32 sums of 8192 products in two orders, then one rounding to bf16 each
        assert ((o.double() - base[k].double()).abs() <= 2.0 ** -7 * base[k].double().abs() + 2.0 ** -12).all()
