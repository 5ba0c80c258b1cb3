"""MXFP4 linears of many tokens on a weight unpacked to bf16: edges of the packed 128 x 128 tiles and of the 256 x 256 output tiles, every
post-op, scratch too small for the unpacked weight. References in 64 bits on the dequantized weight."""
import ctypes

import pytest
import torch

from tests.gpu_util import assert_no_kernel_error, knob_env

pytestmark = pytest.mark.gpu

# tokens, features, inner size
SHAPES = [(129, 32, 64), (256, 160, 192), (300, 288, 1536), (515, 4096, 320), (1030, 2080, 2048), (2050, 1312, 448)]


def _rnd(g, *s, std=1.0):
    return (torch.randn(*s, generator=g, device="cuda") * std).to(torch.bfloat16)


def _weight(g, N, K):
    w = _rnd(g, N, K, std=K ** -0.5)
    w[0, :32] = 0  # an empty block
    w[-1] *= 2.0 ** -40
    q, code, scale = _quantize(w)
    return q, (code * scale).view(N, K)


def _quantize(w):
    """The packed weight, and its codes and scales in float64 [N, K / 32, 32], [N, K / 32, 1]."""
    from tpp_pytorch_extension_b200.llm.llm_common import quantize_weight
    N = w.shape[0]
    q = quantize_weight(w, "mxfp4")
    b = w.double().view(N, -1, 32)
    top = b.abs().amax(-1, keepdim=True)
    scale = torch.where(top > 0, torch.exp2(torch.floor(torch.log2(top.clamp(min=1e-30))) - 2), torch.ones_like(top))
    a = (b / scale).abs()
    step = torch.where(a < 2, 0.5, torch.where(a < 4, 1.0, 2.0))
    return q, torch.sign(b) * (torch.round(a / step) * step).clamp(max=6), scale


def _sum_slack(x, w):
    """What sums of K products in 32 bits may be off by, element by element: the MMAs add sixteen products at a time and may cut a sum's last
    bit, 2^-23 of what has been added up; a few more additions join the pieces of a cut tile."""
    return (x.shape[1] / 16 + 8) * 2.0 ** -23 * (x.double().abs() @ w.abs().T)


def _packed_slack(x, w):
    """The form on the packed weight cuts an activation into two E4M3 terms with one scale per token: what they leave is at most 2^-9 of
    the row's largest value, of either sign."""
    return _sum_slack(x, w) + 2.0 ** -9 * x.double().abs().amax(1, keepdim=True) * w.norm(dim=1)


def _close(got, want, slack):
    """Element by element: half a unit of a bf16 result is at most 2^-8 of it; `slack` is what the value in front of that rounding may be off by."""
    off = (got.double() - want).abs()
    bound = 2.0 ** -8 * (1 + 2.0 ** -10) * (want.abs() + slack) + slack + 1e-45
    assert bool((off <= bound).all()), float((off / bound).max())


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_post_ops(M, N, K):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    q, w = _weight(g, N, K)
    x, bias, mul, res, gamma = _rnd(g, M, K), _rnd(g, N), _rnd(g, M, N), _rnd(g, M, N), _rnd(g, K)
    y = x.double() @ w.T
    h = y + bias.double()
    e = _sum_slack(x, w)
    xn = x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-5) * gamma.double()
    xr = xn.to(torch.bfloat16)
    # a normed value whose rounding is nearly a tie may be rounded the other way (2^-8 of it): about one in 5000, eight in a row allowed
    flips = 8 * 2.0 ** -8 * xn.abs().amax(1, keepdim=True) * w.abs().amax(1)
    silu, fast = h * torch.sigmoid(h), 2.0 ** -20  # of an activation: exponentials and quotients of the special-function unit
    with knob_env(TPX_MXFP4_DENSE=1):
        _close(F.fc_plain(x, q), y, e)
        # slopes of both activations are at most 1.13; h's own 32-bit rounding is in the slack's last additions
        _close(F.fc_plain_act(x, q, bias, "silu", mul, res, 0.5), silu * mul.double() + 0.5 * res.double(),
               (1.2 * (e + 2.0 ** -23 * h.abs()) + fast * silu.abs()) * mul.double().abs() + 2.0 ** -23 * res.double().abs())
        _close(F.fc_plain_act(x, q, bias, "gelu"), torch.nn.functional.gelu(h), 1.2 * (e + 2.0 ** -23 * h.abs()) + fast * h.abs())
        _close(F.fc_plain_norm(x, gamma, 1e-5, q, bias), xr.double() @ w.T + bias.double(), _sum_slack(xr, w) + flips + 2.0 ** -23 * h.abs())
        assert_no_kernel_error()


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gate_up(M, N, K):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    g = torch.Generator(device="cuda").manual_seed(M + N + K + 1)
    (qg, wg), (qu, wu) = _weight(g, N, K), _weight(g, N, K)
    x = _rnd(g, M, K)
    gate, up = x.double() @ wg.T, x.double() @ wu.T
    eg, eu = _sum_slack(x, wg), _sum_slack(x, wu)
    act = gate * torch.sigmoid(gate)
    with knob_env(TPX_MXFP4_DENSE=1):
        _close(F.fc_gate_up(x, qg, qu), act * up, 1.2 * eg * up.abs() + eu * (act.abs() + 1.2 * eg) + 2.0 ** -20 * (act * up).abs())
        _close(F.fc_gate_up(x, qg, qu, "relu"), gate.clamp(min=0) * up, eg * up.abs() + eu * (gate.clamp(min=0) + eg) + 2.0 ** -23 * (gate * up).abs())
        assert_no_kernel_error()


@pytest.mark.parametrize("byte", [0, 1, 2, 3, 127, 252, 253, 254])
@pytest.mark.parametrize("pair", [0, 1])
def test_scales_at_the_ends_of_their_range(byte, pair):
    """Every scale byte is exact, also where a code times its scale is beyond bf16 (253 and 254) or subnormal (0 to 2)."""
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    M, N, K = 300, 256, 512
    g = torch.Generator(device="cuda").manual_seed(byte)
    q, code, _ = _quantize(_rnd(g, N, K))
    q.scales.fill_(byte)
    x = (_rnd(g, M, K).float() * 2.0 ** -max(min(byte - 127, 100), -100)).to(torch.bfloat16)
    y = x.double() @ (code.view(N, K) * 2.0 ** (byte - 127)).T
    with knob_env(TPX_MXFP4_DENSE=1):
        got = F.fc_gate_up(x, q, q, "relu") if pair else F.fc_plain(x, q)
        assert_no_kernel_error()
    assert got.isfinite().all()
    e = _sum_slack(x, code.view(N, K) * 2.0 ** (byte - 127))
    _close(got, y.clamp(min=0) * y if pair else y, 2 * e * (y.abs() + e) if pair else e)


def test_a_block_without_a_value():
    """Scale byte 255 is the format's NaN: every result that its block enters is NaN, whatever the block's codes, and no other is."""
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    M, N, K = 300, 256, 512
    g = torch.Generator(device="cuda").manual_seed(5)
    q, code, scale = _quantize(_rnd(g, N, K).abs())
    x = _rnd(g, M, K).abs()
    w = (code * scale).view(N, K)
    want = x.double() @ w.T
    q.scales.view(N // 32, K // 64, 2, 32)[1, 3, 1, 7] = 255  # feature 39, block 7
    with knob_env(TPX_MXFP4_DENSE=1):
        got = F.fc_plain(x, q)
    bad = torch.zeros_like(got, dtype=torch.bool)
    bad[:, 39] = True
    assert torch.equal(got.isnan(), bad)
    _close(got[~bad], want[~bad], _sum_slack(x, w)[~bad])


@pytest.mark.parametrize("less", [0, 1])
def test_scratch_of_the_packed_form_still_serves(less):
    """A caller that gives only what the form on the packed weight needs gets that form; one byte less is refused."""
    from tpp_pytorch_extension_b200 import _lib
    M, N, K = 300, 512, 512
    g = torch.Generator(device="cuda").manual_seed(3)
    q, w = _weight(g, N, K)
    x, y = _rnd(g, M, K), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    L = _lib.lib()
    with knob_env(TPX_MXFP4_DENSE=0):
        need = L.tpx_qlinear_mxfp4_tc_scratch_bytes(M, N, K, 0)
    with knob_env(TPX_MXFP4_DENSE=1):
        assert L.tpx_qlinear_mxfp4_tc_scratch_bytes(M, N, K, 0) > need
        sc = torch.zeros(need, device="cuda", dtype=torch.uint8)
        wq, sfa = q.packed_tc(None)
        rc = L.tpx_qlinear_mxfp4_tc(wq.data_ptr(), sfa.data_ptr(), 0, x.data_ptr(), M, N, K, None, 0, None, None, ctypes.c_float(1.0), y.data_ptr(),
                                    sc.data_ptr(), need - less, _lib.stream())
        torch.cuda.synchronize()
    assert (rc != 0) == bool(less)
    if not less:
        _close(y, x.double() @ w.T, _packed_slack(x, w))


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_the_unpacked_form_runs(M, N, K, pair):
    """A call that is given the scratch leaves the unpacked weight (a quarter of it; of a pair the rows in turn) there."""
    from tpp_pytorch_extension_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(M + N + K + 2)
    (q, w), (q2, w2) = _weight(g, N, K), _weight(g, N, K)
    x, y = _rnd(g, M, K), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    L = _lib.lib()
    with knob_env(TPX_MXFP4_DENSE=1):
        need = L.tpx_qlinear_mxfp4_tc_scratch_bytes(M, N, K, pair)
        sc = torch.zeros(need, device="cuda", dtype=torch.uint8)
        wq, sfa = q.packed_tc(q2 if pair else None)
        _lib.check(L.tpx_qlinear_mxfp4_tc(wq.data_ptr(), sfa.data_ptr(), pair, x.data_ptr(), M, N, K, None, 0, None, None, ctypes.c_float(1.0), y.data_ptr(),
                                          sc.data_ptr(), need, _lib.stream()))
    rows = (torch.stack([w, w2], 1).view(2 * N, K) if pair else w).mul(0.25).to(torch.bfloat16).flatten()
    held = (sc[at:at + 2 * rows.numel()].view(torch.bfloat16) for at in range(65536, need - 2 * rows.numel() + 1, 1024))
    assert any(torch.equal(h, rows) for h in held if torch.equal(h[64:128], rows[64:128]))  # (equal as values: zeros have two signs)


def test_pinned_host_input_of_many_tokens():
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    M, N, K = 4100, 256, 512
    g = torch.Generator(device="cuda").manual_seed(4)
    q, w = _weight(g, N, K)
    x = _rnd(g, M, K)
    out = torch.empty(M, N, dtype=torch.bfloat16, pin_memory=True)
    F.fc_plain(x.cpu().pin_memory(), q, out=out)
    torch.cuda.synchronize()
    _close(out.cuda(), x.double() @ w.T, _packed_slack(x, w))
