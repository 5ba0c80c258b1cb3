"""MXFP4 linears of many tokens on a weight unpacked to bf16: edges of the packed 128 x 128 tiles and of the 256 x 256 output tiles, every
post-op, scratch too small for the unpacked weight. References in 64 bits on the dequantized weight."""
import ctypes

import pytest
import torch

from tests.gpu_util import assert_no_kernel_error, knob_env

pytestmark = pytest.mark.gpu

# tokens, features, inner size
SHAPES = [(129, 32, 64), (256, 160, 192), (300, 288, 1536), (515, 4096, 320), (1030, 2080, 2048), (2050, 1312, 448)]
TOL = 2.0 ** -8  # rounded to bf16 once, 2^-9 of the value; the rest for sums in 32 bits


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


def _close(got, want):
    assert float((got.double() - want).abs().max()) <= TOL * float(want.abs().max())


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_post_ops(M, N, K):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    q, w = _weight(g, N, K)
    x, bias, mul, res, gamma = _rnd(g, M, K), _rnd(g, N), _rnd(g, M, N), _rnd(g, M, N), _rnd(g, K)
    y = x.double() @ w.T
    h = y + bias.double()
    xn = x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-5) * gamma.double()
    with knob_env(TPX_MXFP4_DENSE=1):
        _close(F.fc_plain(x, q), y)
        _close(F.fc_plain_act(x, q, bias, "silu", mul, res, 0.5), h * torch.sigmoid(h) * mul.double() + 0.5 * res.double())
        _close(F.fc_plain_act(x, q, bias, "gelu"), torch.nn.functional.gelu(h))
        _close(F.fc_plain_norm(x, gamma, 1e-5, q, bias), xn.to(torch.bfloat16).double() @ w.T + bias.double())
        assert_no_kernel_error()


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gate_up(M, N, K):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    g = torch.Generator(device="cuda").manual_seed(M + N + K + 1)
    (qg, wg), (qu, wu) = _weight(g, N, K), _weight(g, N, K)
    x = _rnd(g, M, K)
    gate, up = x.double() @ wg.T, x.double() @ wu.T
    with knob_env(TPX_MXFP4_DENSE=1):
        _close(F.fc_gate_up(x, qg, qu), gate * torch.sigmoid(gate) * up)
        _close(F.fc_gate_up(x, qg, qu, "relu"), gate.clamp(min=0) * up)
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
    _close(got, y.clamp(min=0) * y if pair else y)


def test_a_block_without_a_value():
    """Scale byte 255 is the format's NaN: every result that its block enters is NaN, whatever the block's codes, and no other is."""
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    M, N, K = 300, 256, 512
    g = torch.Generator(device="cuda").manual_seed(5)
    q, code, scale = _quantize(_rnd(g, N, K).abs())
    x = _rnd(g, M, K).abs()
    want = x.double() @ (code * scale).view(N, K).T
    q.scales.view(N // 32, K // 64, 2, 32)[1, 3, 1, 7] = 255  # feature 39, block 7
    with knob_env(TPX_MXFP4_DENSE=1):
        got = F.fc_plain(x, q)
    bad = torch.zeros_like(got, dtype=torch.bool)
    bad[:, 39] = True
    assert torch.equal(got.isnan(), bad)
    _close(got[~bad], want[~bad])


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
        _close(y, x.double() @ w.T)


def test_pinned_host_input_of_many_tokens():
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    M, N, K = 4100, 256, 512
    g = torch.Generator(device="cuda").manual_seed(4)
    q, w = _weight(g, N, K)
    x = _rnd(g, M, K)
    out = torch.empty(M, N, dtype=torch.bfloat16, pin_memory=True)
    F.fc_plain(x.cpu().pin_memory(), q, out=out)
    torch.cuda.synchronize()
    _close(out.cuda(), x.double() @ w.T)
