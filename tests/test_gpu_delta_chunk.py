"""Generalized delta rule in chunks of sixteen tokens: whole and cut last chunks, padding in front, a state to start from, calls in portions, decays at their
ends. Reference: the recurrence token by token in 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
H, D, EPS = 3, 64, 1e-6


def _call(proj, wraw, bias, norm, state, start):
    from tpp_pytorch_extension_b200 import _lib
    B, S, _ = wraw.shape
    out = torch.zeros(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    raw = torch.empty(B * S, H * D, device="cuda")
    a = _lib.DeltaRuleStruct(proj=proj.data_ptr(), wraw=wraw.data_ptr(), a_bias=bias.data_ptr(), norm_w=norm.data_ptr(), start=start.data_ptr(), dev_len=None,
                             state=state.data_ptr(), raw=raw.data_ptr(), out=out.data_ptr(), B=B, S=S, past=0, ldp=5 * H * D, ldo=H * D, heads=H, dim=D, eps=EPS, f32=0)
    _lib.check(_lib.lib().tpx_delta_rule(ctypes.byref(a), _lib.stream()))
    return out.view(B, S, H * D)


def _reference(proj, wraw, bias, norm, state, start):
    B, S, _ = wraw.shape
    r, k, v, a, g = (proj.double().view(B, S, 5, H, D)[:, :, i] for i in range(5))
    w = torch.exp(-torch.exp(torch.tensor(-0.5, dtype=torch.float64)).cuda() * torch.sigmoid(wraw.double().view(B, S, H, D)))
    a = torch.sigmoid(a + bias.double().view(H, D))
    u = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    s, out = state.double().clone(), torch.zeros_like(v)
    for b in range(B):
        for t in range(int(start[b]), S):
            s[b] = w[b, t].unsqueeze(-1) * s[b] - (a[b, t] * u[b, t]).unsqueeze(-1) * (u[b, t].unsqueeze(-2) @ s[b]) + k[b, t].unsqueeze(-1) * v[b, t].unsqueeze(-2)
            o = (r[b, t].unsqueeze(-2) @ s[b]).squeeze(-2)
            out[b, t] = o * torch.rsqrt((o * o).mean(-1, keepdim=True) + EPS) * norm.double().view(H, D) * torch.sigmoid(g[b, t])
    return out.reshape(B, S, H * D), s


@pytest.mark.parametrize("S", [32, 33, 47, 48, 49, 130])
@pytest.mark.parametrize("decay", [0.0, 12.0, -12.0])
def test_against_the_recurrence(S, decay):
    B = 3
    g = torch.Generator(device="cuda").manual_seed(S)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    proj, wraw = rnd(B, S, 5 * H * D).to(torch.bfloat16), rnd(B, S, H * D) * 2 + decay  # decays about their middle, exp(-e^(-1/2)) and 1
    bias, norm, state = rnd(H * D), 1 + 0.1 * rnd(H * D), rnd(B, H, D, D)
    start = torch.tensor([0, 5, S - 1], dtype=torch.int32, device="cuda")
    want, end = _reference(proj, wraw, bias, norm, state, start)
    got = state.clone()
    out = _call(proj, wraw, bias, norm, got, start)
    # a token's decay and rate are right to 2^-21 (exponential, sigmoid, their products), its update is rounded a few times; all of it may stay in the state
    tol = (S + 16) * 2.0 ** -21
    assert float((got.double() - end).norm() / end.norm()) < tol
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -9 + tol
    for b in range(B):
        assert not out[b, :int(start[b])].any()
    # the same in two calls
    part, cut = state.clone(), 32 if S > 64 else S // 2
    zero = torch.zeros_like(start)
    first = _call(proj[:1, :cut].contiguous(), wraw[:1, :cut].contiguous(), bias, norm, part[:1], zero)
    second = _call(proj[:1, cut:].contiguous(), wraw[:1, cut:].contiguous(), bias, norm, part[:1], zero)
    assert float((part[0].double() - end[0]).norm() / end[0].norm()) < tol
    assert float((torch.cat([first, second], 1).double() - want[:1]).norm() / want[:1].norm()) < 2.0 ** -9 + tol
