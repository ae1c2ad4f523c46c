"""Scores that are not finite: a row that sees a NaN or a +inf score comes out NaN, whichever column of a sub-block the
score falls on (the kernels compute part of a row's exponentials with a polynomial that clamps its argument), and no
other row changes."""
import pytest
import torch

from kernelfuser_b200.api import attention_forward, check_status

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,hq,variant", [(128, 2, 1), (128, 2, 2), (128, 2, 3), (128, 2, 5),
                                          (256, 2, 2), (256, 2, 3), (256, 3, 3)])
@pytest.mark.parametrize("first", [0, 64, 128])  # sub-block: a row's first, an ordinary one, a masked one
@pytest.mark.parametrize("score,causal", [("nan", False), ("inf", False), ("nan", True), ("inf", True)])
def test_one_bad_key_spoils_the_rows_that_see_it(D, hq, variant, first, score, causal):
    B, S = 64, 192  # batch element b holds its bad key in column b of the sub-block
    g = torch.Generator(device="cuda").manual_seed(11)
    q, k, v = (torch.randn(B, h, S, D, generator=g, device="cuda", dtype=torch.bfloat16) for h in (hq, 1, 1))
    q[..., 0] = 1.0

    def run(keys):
        out = torch.empty_like(q)
        attention_forward(q, keys, v, None, None, None, out, causal=causal, fuse_q=False, variant=variant)
        torch.cuda.synchronize()
        check_status()
        return out

    clean, bad = run(k), k.clone()
    b = torch.arange(B, device="cuda")
    bad[b, 0, first + b] = 0.0
    bad[b, 0, first + b, 0] = float(score)
    out = run(bad)
    sees = (torch.arange(S, device="cuda")[None] >= first + b[:, None]) if causal else torch.ones(
        B, S, dtype=torch.bool, device="cuda")
    sees = sees[:, None, :, None].expand_as(out)
    assert torch.isnan(out[sees]).all(), int((~torch.isnan(out) & sees).sum())
    assert torch.equal(out[~sees], clean[~sees])
