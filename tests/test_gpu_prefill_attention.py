"""Prefill attention on the tensor cores where its softmax takes different ways: scores of any size, and masks that touch some of a tile's
groups of 32 keys and not others. Reference in 64 bits."""
import pytest
import torch

from tests.gpu_util import assert_no_kernel_error

pytestmark = pytest.mark.gpu


def _case(H, S, grow, padding, dropped):
    """B = 2, two kv heads, two queries per key head. Every token's query is its own key times 2^grow, so that its own score stands out;
    padding: keys dropped in front of the second sequence; dropped: single keys dropped in both."""
    from tpp_pytorch_extension_b200._C._tpp_attn import attention
    B, N, R = 2, 2, 2
    g = torch.Generator(device="cuda").manual_seed(H + S + grow + padding + len(dropped))
    k, v = (torch.randn(B, N, S, H, generator=g, device="cuda").bfloat16() for _ in range(2))
    q = (k.unsqueeze(3).expand(B, N, S, R, H).float() * 2.0 ** grow).bfloat16().contiguous()
    blocks = (S + 31) // 32 + 4
    kc, vc = (torch.zeros(blocks * 32, B, N, H, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    kc[:S], vc[:S] = k.permute(2, 0, 1, 3), v.permute(2, 0, 1, 3)
    kc, vc = (t.view(blocks, 32, B, N, H).permute(0, 2, 3, 1, 4).contiguous() for t in (kc, vc))
    mask = torch.zeros(B, (S + 31) // 32 * 32, device="cuda", dtype=torch.bfloat16)
    mask[1, :padding] = torch.finfo(torch.bfloat16).min
    mask[:, dropped] = torch.finfo(torch.bfloat16).min
    got = attention(q, kc, vc, mask if padding or dropped else None, S).double()
    assert_no_kernel_error()
    score = torch.einsum("bnsrh,bnth->bnsrt", q.double(), k.double()) * H ** -0.5 + mask[:, None, None, None, :S].double()
    score = score.masked_fill(torch.ones(S, S, device="cuda").triu(1).bool()[:, None], -float("inf"))
    want = torch.einsum("bnsrt,bnth->bnsrh", score.softmax(-1), v.double())
    real = torch.ones(B, S, dtype=torch.bool, device="cuda")  # tokens that are dropped themselves have no score that stands out
    real[1, :padding] = False
    real[:, dropped] = False
    keep = real[:, None, :, None, None].expand_as(got)
    # weights (which sum to one) and the result are rounded to bf16 once each: at most 2^-8 of max |v| each
    assert float((got - want)[keep].abs().max()) <= 2.0 ** -7 * float(v.double().abs().max())


@pytest.mark.parametrize("grow", [0, 8, 13, 29, 31, 60, 110])
@pytest.mark.parametrize("H,S", [(128, 300), (64, 129)])
def test_scores_of_any_size(H, S, grow):
    _case(H, S, grow, 0, [])


@pytest.mark.parametrize("grow", [0, 29])
@pytest.mark.parametrize("padding,dropped", [(5, []), (32, []), (150, []), (0, [70]), (0, [31, 128, 200]), (33, [64])])
@pytest.mark.parametrize("H,S", [(128, 300), (64, 257)])
def test_masks_that_touch_some_groups_of_keys(H, S, padding, dropped, grow):
    _case(H, S, grow, padding, dropped)
