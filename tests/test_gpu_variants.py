"""Every attention kernel variant (baseline, pipelined, persistent, one tile per CTA) against the
FP32 oracle on the same inputs; the default (automatic) choice is covered by
tests/test_gpu_attention.py."""
import pytest
import torch

import kernelfuser_b200 as kf
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [1, 2, 3, 5])
@pytest.mark.parametrize("s,hq,hkv,causal,dtype", [
    (517, 8, 2, True, torch.bfloat16),    # even GQA group: two heads per CTA, ragged tail
    (390, 6, 2, True, torch.float16),     # odd group size: two query blocks of one head per CTA
    (129, 3, 3, False, torch.bfloat16),   # G = 1, second tile of the last pair is empty
    (64, 4, 4, True, torch.bfloat16),     # a single sub-block
])
def test_variant_matches_oracle(variant, s, hq, hkv, causal, dtype):
    # one seed for all variants: every kernel sees the same rows, so a difference
    # between variants is a difference between kernels, not between inputs
    xs = kf.make_inputs(3, s, hq, hkv, 128, dtype=dtype, seed=41)
    ref = orc.oracle_fp32(*xs, causal)
    out = kf.optimized_attention(*[x.cuda() for x in xs], causal=causal, variant=variant)
    torch.cuda.synchronize()
    kf.check_status()
    m = orc.metric(out.cpu(), ref)
    assert orc.within_tolerance(m), (variant, s, hq, hkv, m)


def test_many_items_per_persistent_cta():
    # more work items than SMs, so every CTA of the persistent kernel walks several items
    xs = kf.make_inputs(6, 700, 16, 4, 128, seed=77)
    ref = orc.oracle_fp32(*xs, True)
    dx = [x.cuda() for x in xs]
    outs = [kf.optimized_attention(*dx, causal=True, variant=v) for v in (3, 1)]
    torch.cuda.synchronize()
    kf.check_status()
    for o in outs:
        assert orc.within_tolerance(orc.metric(o.cpu(), ref))


def test_d128_only_variants_reject_d256():
    xs = [x.cuda() for x in kf.make_inputs(1, 64, 2, 1, 256, seed=1)]
    for variant in (5,):
        with pytest.raises(ValueError):
            kf.optimized_attention(*xs, causal=True, variant=variant)


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("s,hq,hkv,causal,dtype", [
    (517, 4, 2, True, torch.bfloat16),
    (200, 3, 1, False, torch.float16),
    (64, 2, 2, True, torch.bfloat16),
])
def test_d256_variants_match_oracle(variant, s, hq, hkv, causal, dtype):
    xs = kf.make_inputs(2, s, hq, hkv, 256, dtype=dtype, theta=1e4, seed=61)
    ref = orc.oracle_fp32(*xs, causal)
    out = kf.optimized_attention(*[x.cuda() for x in xs], causal=causal, variant=variant)
    torch.cuda.synchronize()
    kf.check_status()
    m = orc.metric(out.cpu(), ref)
    assert orc.within_tolerance(m), (variant, s, hq, hkv, m)


def test_persistent_kernels_reuse_their_counter_slots():
    # The persistent kernels take work from counters in the library image, slots used in turn and reset by the
    # last CTA of each launch: run launches one behind the other on two streams, both head dims, more of them than
    # there are slots, and compare every result with the first one of its kind.
    xs128 = [x.cuda() for x in kf.make_inputs(2, 640, 8, 2, 128, seed=5)]
    xs256 = [x.cuda() for x in kf.make_inputs(1, 512, 4, 2, 256, theta=1e4, seed=6)]
    ref128 = kf.optimized_attention(*xs128, causal=True, variant=3)
    ref256 = kf.optimized_attention(*xs256, causal=True, variant=3)
    torch.cuda.synchronize()
    kf.check_status()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    outs = []
    for i in range(1100):
        xs, ref = (xs128, ref128) if i % 3 else (xs256, ref256)
        if i % 2:
            with torch.cuda.stream(side):
                outs.append((kf.optimized_attention(*xs, causal=True, variant=3), ref))
        else:
            outs.append((kf.optimized_attention(*xs, causal=True, variant=3), ref))
    torch.cuda.synchronize()
    kf.check_status()
    for out, ref in outs:
        assert torch.equal(out, ref)


@pytest.mark.parametrize("b,s,hq,hkv,causal,dtype", [
    (1, 1, 2, 1, True, torch.bfloat16),     # one row, one pair of CTAs
    (3, 65, 4, 2, False, torch.float16),    # the second sub-block has one key: CTA 1's half of it lies past the end
    (2, 97, 4, 1, True, torch.bfloat16),    # ... and starts there
    (16, 300, 16, 4, True, torch.bfloat16), # several items per pair of CTAs, ragged tail
    (20, 129, 8, 4, False, torch.float16),  # items of three sub-blocks: shorter than the claim distance
])
def test_d256_sm_pairs_match_oracle(b, s, hq, hkv, causal, dtype):
    xs = kf.make_inputs(b, s, hq, hkv, 256, dtype=dtype, theta=1e4, seed=67)
    ref = orc.oracle_fp32(*xs, causal)
    out = kf.optimized_attention(*[x.cuda() for x in xs], causal=causal, variant=3)
    torch.cuda.synchronize()
    kf.check_status()
    m = orc.metric(out.cpu(), ref)
    assert orc.within_tolerance(m), (b, s, hq, hkv, m)


@pytest.mark.parametrize("variant,hq,hkv", [(2, 4, 2), (3, 4, 2), (3, 3, 1), (3, 2, 2)])
def test_d256_kernels_drain_on_a_status(variant, hq, hkv):
    # a launch that finds an earlier failure leaves without touching the output; on SM pairs both CTAs follow one reading
    xs = [x.cuda() for x in kf.make_inputs(2, 300, hq, hkv, 256, theta=1e4, seed=68)]
    word = kf.status_word(xs[0].device)
    word.fill_(7)
    out = torch.full_like(xs[0], float("nan"))
    kf.optimized_attention(*xs, causal=True, out=out, variant=variant)
    torch.cuda.synchronize()
    with pytest.raises(kf.KernelStatusError, match="7"):
        kf.check_status()
    assert torch.isnan(out).all()
    again = kf.optimized_attention(*xs, causal=True, out=out, variant=variant)
    torch.cuda.synchronize()
    kf.check_status()
    assert torch.isfinite(again).all()


def device_inputs(b, s, hq, hkv, d, dtype=torch.bfloat16, seed=9):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *shape: torch.randn(*shape, generator=g, device="cuda", dtype=dtype)
    cos, sin = kf.inputs.rope_tables(torch.arange(s, device="cuda"), d, 1e4, dtype)
    return r(b, hq, s, d), r(b, hkv, s, d), r(b, hkv, s, d), 1 + 0.1 * r(d), 1 + 0.1 * r(d), cos, sin


@pytest.mark.parametrize("b,s,hq,hkv,causal,dtype", [
    (16, 300, 12, 4, True, torch.bfloat16),  # 576 tiles: about four for each CTA
    (40, 64, 3, 1, False, torch.float16),    # tiles of one sub-block, shorter than the claim distance, ...
    (80, 64, 3, 3, True, torch.bfloat16),    # ... and more of them than SMs
    (12, 700, 24, 8, True, torch.bfloat16),  # 1728 tiles: only the last groups are interleaved
    (6, 700, 24, 24, False, torch.float16),  # as many KV heads as query heads, no mask
])
def test_d256_one_cta_per_tile_walks_many_tiles(b, s, hq, hkv, causal, dtype):
    # odd numbers of query heads per KV head: the persistent kernel without SM pairs, against one launch item per tile
    xs = device_inputs(b, s, hq, hkv, 256, dtype)
    ref = kf.optimized_attention(*xs, causal=causal, variant=2)
    out = kf.optimized_attention(*xs, causal=causal, variant=3)
    torch.cuda.synchronize()
    kf.check_status()
    assert torch.equal(out, ref)


@pytest.mark.parametrize("b,s,hq,hkv,causal", [
    (4, 1100, 16, 8, True),    # 288 items: about four for each pair
    (24, 700, 16, 8, True),    # 1152 items: only the last groups are interleaved
    (1, 4096, 4, 1, False),    # long items
])
def test_d256_sm_pairs_equal_one_launch_item_per_tile(b, s, hq, hkv, causal):
    # the same sub-blocks in the same order: bit for bit, and the same again
    xs = device_inputs(b, s, hq, hkv, 256)
    ref = kf.optimized_attention(*xs, causal=causal, variant=2)
    outs = [kf.optimized_attention(*xs, causal=causal, variant=3) for _ in range(3)]
    torch.cuda.synchronize()
    kf.check_status()
    assert all(torch.equal(out, ref) for out in outs)


@pytest.mark.parametrize("b,s,hq,hkv,d,variant", [
    (1, 16384, 32, 8, 128, 3),   # a long launch of two-head items
    (2, 4096, 16, 8, 256, 3),    # SM pairs
    (2, 4096, 24, 8, 256, 3),    # one CTA per tile
])
def test_automatic_choice_of_a_long_launch(b, s, hq, hkv, d, variant):
    xs = device_inputs(b, s, hq, hkv, d)
    auto = kf.optimized_attention(*xs, causal=True)
    named = kf.optimized_attention(*xs, causal=True, variant=variant)
    other = kf.optimized_attention(*xs, causal=True, variant=2)
    # a model's layout: projections read in place, the result written as [B, S, Hq*D]
    views = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in xs[:3]]
    flat = kf.fused(*views, *xs[3:], True, out_layout="bshd")
    torch.cuda.synchronize()
    kf.check_status()
    assert torch.equal(auto, named)
    assert torch.equal(auto, other)
    assert torch.equal(flat.view(b, s, hq, d).transpose(1, 2), auto)


@pytest.mark.parametrize("s", [65, 517])
@pytest.mark.parametrize("hq,hkv,d,variant", [(8, 2, 128, 3), (8, 2, 128, 2), (8, 2, 128, 5), (4, 2, 256, 3),
                                              (3, 1, 256, 3), (4, 2, 256, 2)])
def test_every_kernel_reads_and_writes_strided_rows(s, hq, hkv, d, variant):
    # [B,S,H,D] storage for every tensor, and rows of the output that lie further apart than its heads fill
    from kernelfuser_b200.api import attention_forward
    q, k, v, gq, _, cos, sin = device_inputs(2, s, hq, hkv, d)
    want = attention_forward(q, k, v, gq, cos, sin, torch.empty_like(q), causal=True, variant=variant)
    views = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v)]
    store = torch.full((2, s, hq + 1, d), 7.0, dtype=q.dtype, device="cuda")
    out = store[:, :, :hq].transpose(1, 2)
    attention_forward(*views, gq, cos, sin, out, causal=True, variant=variant)
    torch.cuda.synchronize()
    kf.check_status()
    assert torch.equal(out, want)
    assert (store[:, :, hq] == 7.0).all()
