"""Generalized delta rule in chunks of sixteen tokens: whole and cut last chunks, padding in front, a state to start from, calls in portions, decays at their
ends, as many heads as one round of CTAs holds; infinities, NaN and values whose products overflow. References: the recurrence token by token in 64 bits,
and the token loop, which calls of fewer than 32 tokens take."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
H, D, EPS = 3, 64, 1e-6


def _call(proj, wraw, bias, norm, state, start, past=0):
    from tpp_pytorch_extension_b200 import _lib
    B, S, _ = wraw.shape
    H = norm.numel() // D
    out = torch.zeros(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    raw = torch.empty(B * S, H * D, device="cuda")
    a = _lib.DeltaRuleStruct(proj=proj.data_ptr(), wraw=wraw.data_ptr(), a_bias=bias.data_ptr(), norm_w=norm.data_ptr(), start=start.data_ptr(), dev_len=None,
                             state=state.data_ptr(), raw=raw.data_ptr(), out=out.data_ptr(), B=B, S=S, past=past, ldp=5 * H * D, ldo=H * D, heads=H, dim=D, eps=EPS, f32=0)
    _lib.check(_lib.lib().tpx_delta_rule(ctypes.byref(a), _lib.stream()))
    return out.view(B, S, H * D)


def _portions(proj, wraw, bias, norm, state, start, length):
    """The call in portions; those of fewer than 32 tokens go through the token loop."""
    B, S, _ = wraw.shape
    out = [_call(proj.view(B, S, -1)[:, t:t + length].contiguous(), wraw[:, t:t + length].contiguous(), bias, norm, state, start, t) for t in range(0, S, length)]
    return torch.cat(out, 1)


def _reference(proj, wraw, bias, norm, state, start):
    B, S, _ = wraw.shape
    H = norm.numel() // D
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


def _inputs(B, S, H, seed, decay=0.0, rank=D):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    proj = rnd(B, S, 5, H, D)
    if rank < D:  # keys of few directions
        proj[:, :, 1] = torch.einsum("bshr,hrd->bshd", rnd(B, S, H, rank), rnd(H, rank, D)) * rank ** -0.5
    return proj.to(torch.bfloat16), rnd(B, S, H * D) * 2 + decay, rnd(H * D), 1 + 0.1 * rnd(H * D), rnd(B, H, D, D)


# The loop's sums are rounded, those of the matrix products cut off, whose errors have one sign where the terms have: with keys of all directions the state is no
# further off than the loop's (with slow decays nearer), with keys of a few directions and fast decays up to `times` as far.
@pytest.mark.parametrize("S,H,decay,rank,times", [(130, 4, 0.0, D, 1.0), (513, 16, 0.0, D, 1.0), (513, 16, -3.0, D, 0.75), (130, 4, -12.0, D, 0.75), (130, 4, 12.0, D, 1.05),
                                                  (513, 16, -3.0, 4, 1.0), (513, 16, 0.0, 4, 1.2), (1030, 16, 0.0, 1, 1.5), (130, 4, 12.0, 1, 1.5), (130, 4, -12.0, 1, 0.75)])
def test_error_of_the_token_loop(S, H, decay, rank, times):
    proj, wraw, bias, norm, state = _inputs(1, S, H, S + H, decay, rank)
    start = torch.zeros(1, dtype=torch.int32, device="cuda")
    want, end = _reference(proj, wraw, bias, norm, state, start)
    error = lambda a, b: float((a.double() - b).norm() / b.norm())
    chunked, looped = state.clone(), state.clone()
    out, out2 = _call(proj, wraw, bias, norm, chunked, start), _portions(proj, wraw, bias, norm, looped, start, 31)
    assert error(chunked, end) <= times * error(looped, end)
    assert error(out, want) <= 1.002 * error(out2, want)  # both are the result's rounding to bf16


@pytest.mark.parametrize("more", [0, 1])
def test_heads_of_one_round(more):
    H = torch.cuda.get_device_properties(0).multi_processor_count + more  # with one more the token loop
    proj, wraw, bias, norm, state = _inputs(1, 50, H, more)
    start = torch.tensor([3], dtype=torch.int32, device="cuda")
    want, end = _reference(proj, wraw, bias, norm, state, start)
    out = _call(proj, wraw, bias, norm, state, start)
    assert float((state.double() - end).norm() / end.norm()) < 66 * 2.0 ** -21
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -9 + 66 * 2.0 ** -21


def test_padding_behind_cached_tokens():
    S, past = 40, 100
    proj, wraw, bias, norm, state = _inputs(3, S, 2, 1)
    start = torch.tensor([7, past + 9, past + S + 5], dtype=torch.int32, device="cuda")  # cached already, inside the call, behind it
    want, end = _reference(proj, wraw, bias, norm, state, (start - past).clamp(0, S))
    got = state.clone()
    out = _call(proj, wraw, bias, norm, got, start, past)
    assert float((got.double() - end).norm() / end.norm()) < 56 * 2.0 ** -21
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -9 + 56 * 2.0 ** -21
    assert torch.equal(got[2], state[2])


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf"), 2.0 ** 70, -2.0 ** 120])
@pytest.mark.parametrize("at", [0, 37, 69])
def test_infinity_and_nan(value, at):
    """One such value in r, k, v, a, the gate, the decay and the incoming state, each in a head of its own, the last head without: what the token loop makes of it."""
    B, S, H = 2, 70, 8
    proj, wraw, bias, norm, state = _inputs(B, S, H, 5)
    start = torch.zeros(B, dtype=torch.int32, device="cuda")
    clean, end = state.clone(), state.clone()
    before = _call(proj, wraw, bias, norm, clean, start)
    for i in range(5):
        proj[1, at, i, i, 11] = value
    wraw.view(B, S, H, D)[1, at, 5, 11] = value
    end[1, 6, 11, 13] = value
    looped = end.clone()
    out = _call(proj, wraw, bias, norm, end, start)
    want = _portions(proj, wraw, bias, norm, looped, start, 31)
    for a, b in ((out, want), (end, looped)):
        assert torch.equal(a.isnan(), b.isnan())
        assert torch.equal(a.isinf(), b.isinf())
        # values beside a large one are what its size leaves of them
        a, b = (z.double().nan_to_num(0, 0, 0).view(-1, H, D) if z is not end and z is not looped else z.double().nan_to_num(0, 0, 0).flatten(0, 1) for z in (a, b))
        assert bool(((a - b).norm(dim=-1) <= 2.0 ** -7 * b.norm(dim=-1)).all())
    if value != value:  # from the token on, in no other head, and never turned into a number
        out, before = out.view(B, S, H, D), before.view(B, S, H, D)
        for i in (0, 1, 2, 3, 5):
            assert bool(out[1, at, i].isnan().any())
        for i in (1, 2, 3, 5):
            assert bool(end[1, i].isnan().any()) and bool(out[1, at:, i].isnan().any(-1).all())
        assert bool(out[1, :, 6].isnan().any(-1).all()) and bool(end[1, 6].isnan().any())
        assert not out[1, :at, :6].isnan().any()
        assert torch.equal(out[0], before[0]) and torch.equal(out[1, :, 7], before[1, :, 7])
        assert torch.equal(end[0], clean[0]) and torch.equal(end[1, 7], clean[1, 7])
