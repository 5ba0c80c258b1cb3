"""The many-row linears on CTA pairs (bf16, and 32-bit from bf16 terms): edges of their 256 x 256 tiles, cut tiles, every epilogue, and
values that cannot be cut into terms. References in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows, features, inner size: one tile, tile edges, several tiles with and without a cut along k, an inner size off the k step
SHAPES = [(129, 256, 1024), (256, 512, 4096), (257, 264, 72), (300, 4096, 1536), (1030, 2056, 2048), (2049, 1288, 520), (4100, 5128, 256)]
# a result is rounded to bf16 once: at most 2^-8 of it; in fp32 the sum of K products is off by a few 2^-24 of its size
BF16, F32 = 2.0 ** -8, 2e-6


def _hl():
    from tpp_pytorch_extension_b200._C import _hybrid_layers
    return _hybrid_layers


def _rnd(g, *s, std=1.0, dtype=torch.float32):
    return (torch.randn(*s, generator=g, device="cuda") * std).to(dtype)


def _err(got, want):
    return float((got.double() - want).abs().max() / want.abs().max())


def _gen(*s):
    return torch.Generator(device="cuda").manual_seed(sum(s))


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, BF16), (torch.float32, F32)])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_activation_from_a_column(M, N, K, dtype, tol):
    g, HL = _gen(M, N, K), _hl()
    x, w, b = _rnd(g, M, K + 8, dtype=dtype)[:, :K], _rnd(g, N, K, std=K ** -0.5, dtype=dtype), _rnd(g, N)
    want = x.double() @ w.double().T + b.double()
    want[:, 128:] = torch.tanh(want[:, 128:])
    assert _err(HL.linear(x, w, b, act="tanh", act_from=128), want) < tol
    assert _err(HL.linear(x, w, b, act="tanh", act_from=128, out_f32=True), want) < (tol if dtype is torch.float32 else 1e-5)


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, BF16), (torch.float32, F32)])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gated_units(M, N, K, dtype, tol):
    g, HL = _gen(M, N, K), _hl()
    x, w, b = _rnd(g, M, K, dtype=dtype), _rnd(g, N, K, std=K ** -0.5, dtype=dtype), _rnd(g, N)
    units = (N - 64) // 2
    cat = torch.zeros(M, (16 + units + 7) // 8 * 8, device="cuda", dtype=dtype)
    y = HL.linear_glu(x, w, b, 64, 1.5, cat[:, 16:])
    full = x.double() @ w.double().T + b.double()
    gate, up = full[:, 64::2].clamp(max=1.5), full[:, 65::2].clamp(-1.5, 1.5)
    assert _err(y, full[:, :64]) < tol
    assert _err(cat[:, 16:16 + units], gate * torch.sigmoid(1.702 * gate) * (up + 1)) < 2 * tol
    assert not cat[:, :16].any() and not cat[:, 16 + units:].any()


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, BF16), (torch.float32, F32)])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_stream_and_norm(M, N, K, dtype, tol):
    g, HL = _gen(M, N, K), _hl()
    x, w, res, add = _rnd(g, M, K, dtype=dtype), _rnd(g, N, K, std=K ** -0.5, dtype=dtype), _rnd(g, M, N), _rnd(g, N)
    nw, nb = _rnd(g, N), _rnd(g, N)
    x_out, h = HL.linear_residual(x, w, res, add, (0.5, nw, nb))
    want = res.double() + x.double() @ w.double().T + add.double()
    assert _err(x_out, want) < (tol if dtype is torch.float32 else 1e-5)
    assert _err(h, torch.tanh(0.5 * want) * nw.double() + nb.double()) < tol


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_plain_with_residual_and_multiplier(M, N, K):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    bf = torch.bfloat16
    g = _gen(M, N, K)
    x, w, b, mul, res = (_rnd(g, *s, dtype=bf) for s in ((M, K), (N, K), (N,), (M, N), (M, N)))
    w = (w.float() * K ** -0.5).to(bf)
    want = torch.nn.functional.silu(x.double() @ w.double().T + b.double()) * mul.double() + 0.5 * res.double()
    assert _err(F.fc_plain_act(x, w, b, "silu", mul, res, 0.5), want) < BF16
    # twice the same: the pieces of a cut tile are added in a fixed order
    assert torch.equal(F.fc_plain_act(x, w, b, "silu", mul, res, 0.5), F.fc_plain_act(x, w, b, "silu", mul, res, 0.5))


def _linear_f32(x, w, scratch_bytes):
    """tpx_linear with a scratch of the caller's size: below what the tensor-core form asks for it runs on the CUDA cores."""
    from tpp_pytorch_extension_b200 import _lib
    y = torch.empty(x.shape[0], w.shape[0], device="cuda")
    sc = torch.zeros(scratch_bytes, dtype=torch.uint8, device="cuda")
    _hl()._call("tpx_linear", _lib.LinearStruct(w=w.data_ptr(), x=x.data_ptr(), y=y.data_ptr(), M=x.shape[0], N=w.shape[0], K=x.shape[1], ldw=w.stride(0),
                                                ldx=x.stride(0), ldy=y.stride(0), f32=1, out_f32=1, scratch=sc.data_ptr(), scratch_bytes=scratch_bytes))
    return y


@pytest.mark.parametrize("spread", [0.0, 4.0])  # rows of one size; sizes over many powers of two
@pytest.mark.parametrize("M,N,K", [(64, 2048, 4096), (300, 4096, 1536), (513, 2048, 10240), (2100, 1024, 512)])
def test_f32_terms_lose_nothing(M, N, K, spread):
    from tpp_pytorch_extension_b200 import _lib
    g = _gen(M, N, K)
    x, w = (_rnd(g, *s) * torch.exp2(torch.round(spread * _rnd(g, *s))) for s in ((M, K), (N, K)))
    nb = _lib.lib().tpx_linear_f32_scratch_bytes(M, N, K)
    assert nb > 0
    want = x.double() @ w.double().T
    terms, plain = _linear_f32(x, w, nb), _linear_f32(x, w, 65536)
    off = [float((t.double() - want).norm() / want.norm()) for t in (terms, plain)]
    assert off[0] <= off[1] and off[0] < 1e-6


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("where", ["x", "w", "w_last"])
def test_f32_values_without_terms(bad, where):
    from tpp_pytorch_extension_b200 import _lib
    M, N, K = 200, 9000, 2048  # three slabs of weight rows
    g = _gen(M, N, K)
    x, w = _rnd(g, M, K), _rnd(g, N, K)
    if where == "x":
        x[7, 5] = bad
    else:
        w[3 if where == "w" else N - 1, 5] = bad
    nb = _lib.lib().tpx_linear_f32_scratch_bytes(M, N, K)
    terms, plain = _linear_f32(x, w, nb), _linear_f32(x, w, 65536)
    assert torch.equal(torch.isnan(terms), torch.isnan(plain))
    assert torch.equal(terms.isposinf(), plain.isposinf()) and torch.equal(terms.isneginf(), plain.isneginf())
    fine = plain.isfinite()
    assert torch.allclose(terms[fine], plain[fine], rtol=1e-3, atol=1e-3)


@pytest.mark.parametrize("a,b", [(-112, 0), (-118, 10), (-126, 30), (-130, 60), (-140, 100), (0, -120), (-60, -62), (24, 24), (29, -140)])
def test_f32_operands_of_any_size(a, b):
    """Rows whose values are all near 2^a against weights near 2^b, down to subnormal ones: no further off than the CUDA cores."""
    from tpp_pytorch_extension_b200 import _lib
    M, N, K = 256, 1024, 2048
    g = torch.Generator(device="cuda").manual_seed(a * 1000 + b + 200000)
    x, w = (_rnd(g, *s, dtype=torch.float64).clamp(-1.9, 1.9) * 2.0 ** e for s, e in (((M, K), a), ((N, K), b)))
    x, w = x.float(), w.float()
    want = x.double() @ w.double().T
    off = [float((_linear_f32(x, w, n).double() - want).norm() / want.norm()) for n in (_lib.lib().tpx_linear_f32_scratch_bytes(M, N, K), 65536)]
    assert off[0] <= off[1] < 1e-5


@pytest.mark.parametrize("u,v", [(3e38, 1e3), (-3e38, 1e3), (3e38, -1e30), (2.9e35, 1e9), (1.1e30, 3e12), (2.0 ** 30, 3e38)])
def test_f32_products_beyond_the_range(u, v):
    """Finite operands whose product overflows by any amount: infinities and NaN as on the CUDA cores, whatever the signs of the terms."""
    from tpp_pytorch_extension_b200 import _lib
    M, N, K = 200, 9000, 2048
    g = _gen(M, N, K)
    x, w = _rnd(g, M, K), _rnd(g, N, K)
    x[7, 5], w[3, 5], w[N - 1, 5] = u, v, -v
    x[8, 6], w[4, 6] = u * 0.9, v * 1.01  # other remainders
    terms, plain = _linear_f32(x, w, _lib.lib().tpx_linear_f32_scratch_bytes(M, N, K)), _linear_f32(x, w, 65536)
    assert plain.isinf().any()
    assert torch.equal(terms.isnan(), plain.isnan())
    assert torch.equal(terms.isposinf(), plain.isposinf()) and torch.equal(terms.isneginf(), plain.isneginf())
    fine = plain.isfinite()
    assert torch.allclose(terms[fine], plain[fine], rtol=1e-3, atol=1e-3)
