"""Rows whose maximum climbs along the keys: the exponent base of the pipelined kernels has to move, once or many
times, by a little more than its threshold or by far, in full, masked and ragged sub-blocks.  Compared with the
baseline kernel (variant 1), which takes every block's maximum first."""
import pytest
import torch

import kernelfuser_b200 as kf

pytestmark = pytest.mark.gpu


def climbing(S, D, gain, dtype, hq=4, hkv=2, seed=5):
    """Queries along one direction, keys whose component along it grows with the position: with weights of `gain`
    the scores of a row climb by up to 2 * gain^2 * sqrt(D) over its keys."""
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g)
    u = r(D)
    w = torch.linspace(-3, 3, S)[None, None, :, None]
    q, k, v = r(2, hq, S, D) * 0.5 + u, r(2, hkv, S, D) + w * u, r(2, hkv, S, D)
    gamma = torch.full((D,), gain)
    return [t.to(dtype).cuda() for t in (q, k, v, gamma, gamma)]


@pytest.mark.parametrize("D,variant,hq", [(128, 2, 4), (128, 3, 4), (128, 3, 2), (128, 5, 4), (256, 2, 4), (256, 3, 4),
                                          (256, 3, 2)])  # two KV heads: SM pairs at D = 256 with four query heads only
@pytest.mark.parametrize("S,gain,causal,dtype", [
    (65, 1.0, True, torch.bfloat16),     # one full sub-block and one key
    (700, 1.0, False, torch.float16),    # the base just leaves its threshold
    (700, 3.0, True, torch.bfloat16),    # a move in most sub-blocks, masked ones among them
    (1030, 10.0, False, torch.bfloat16), # scores far above any polynomial's range in a sub-block
])
def test_moving_base_matches_baseline(D, variant, hq, S, gain, causal, dtype):
    q, k, v, gq, gk = climbing(S, D, gain, dtype, hq)
    run = lambda val, var: kf.optimized_attention(q, k, val, gq, gk, causal=causal, variant=var).float()
    ref, out = run(v, 1), run(v, variant)
    weight = run(v.abs(), 1)  # sum of p |v|
    torch.cuda.synchronize()
    kf.check_status()
    # Each kernel rounds the probabilities and the output to 16 bits (half a place each); the polynomial adds 7.5e-5, and
    # fp16 probabilities below 2^-14 of the base, which may lie 2^8 under the maximum, half a subnormal place each.
    # Scores of up to L (|q| |k| scale log2 e, rows of RMS `gain`) are sums of D products in 32 bits, in an order of each
    # kernel's own: D 2^-24 L at most, times ln 2 as a relative error of a probability.
    half = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    tiny = 0.0 if dtype == torch.bfloat16 else 2 * S * 2.0 ** -25 * float(v.abs().max())
    order = 2 * 0.6932 * D * 2.0 ** -24 * 1.4427 * D ** 0.5 * gain ** 2
    bound = (4 * half + 2 * 7.5e-5 + order) * weight * 1.01 + tiny + 1e-6
    worst = float(((out - ref).abs() / bound).max())
    assert torch.isfinite(out).all() and worst <= 1.0, (worst, float((out - ref).abs().max()))
