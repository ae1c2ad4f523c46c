"""Captured launches of the persistent kernels (which take their work from a counter in device memory): a replay may run
next to other replays and to eager calls, on any stream, however many launches lie between the captures."""
import pytest
import torch

import kernelfuser_b200 as kf

pytestmark = pytest.mark.gpu

# more work items than fit the GPU at a time: two tiles per CTA, SM pairs, one CTA per tile
KINDS = [(4, 1024, 16, 4, 128), (4, 1024, 8, 4, 256), (4, 1024, 6, 2, 256)]


def inputs(b, s, hq, hkv, d, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *shape: torch.randn(*shape, generator=g, device="cuda", dtype=torch.bfloat16)
    return r(b, hq, s, d), r(b, hkv, s, d), r(b, hkv, s, d), 1 + 0.1 * r(d), 1 + 0.1 * r(d)


def captured(xs, launches=1):
    out, kn = torch.empty_like(xs[0]), torch.empty_like(xs[1])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for _ in range(launches):
            kf.optimized_attention(*xs, causal=True, variant=3, out=out, kn=kn)
    return g, out, kn  # (the graph writes both: they have to outlive it)


@pytest.mark.parametrize("kind", KINDS)
def test_replays_and_eager_calls_run_next_to_one_another(kind):
    a, b, e = (inputs(*kind, seed=s) for s in (1, 2, 3))
    want = [kf.optimized_attention(*xs, causal=True, variant=2) for xs in (a, b, e)]
    kf.optimized_attention(*a, causal=True, variant=3)
    torch.cuda.synchronize()
    ga, out_a, _kn_a = captured(a)
    for _ in range(63):  # so that counters taken in turns of 64 would meet again
        kf.optimized_attention(*e, causal=True, variant=3)
    gb, out_b, _kn_b = captured(b)
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(20):
        out_a.zero_(), out_b.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(sa):
            ga.replay()
        with torch.cuda.stream(sb):
            gb.replay()
        eager = kf.optimized_attention(*e, causal=True, variant=3)
        torch.cuda.synchronize()
        assert torch.equal(out_a, want[0]) and torch.equal(out_b, want[1]) and torch.equal(eager, want[2])
    kf.check_status()


def test_more_captured_launches_than_counters():
    # the counters of a graph come back when it is destroyed; a launch that finds none runs a kernel without one
    xs = inputs(1, 64, 2, 1, 128, seed=4)
    want = kf.optimized_attention(*xs, causal=True, variant=2)
    for _ in range(2):
        g, out, kn = captured(xs, launches=17000)
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        g.reset()
        del g
    again, out, kn = captured(xs)
    again.replay()
    torch.cuda.synchronize()
    kf.check_status()
    assert torch.equal(out, want)
