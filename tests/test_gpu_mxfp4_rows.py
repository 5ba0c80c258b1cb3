"""MXFP4 linear of few tokens at the edges of its splits: tiles per CTA, the last CTA's overlap, clusters, half and missing k steps, groups of tokens,
who converts the activations; every scale byte; activations from 2^-40 to 2^40 and infinities; a recorded chain. Reference: 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

E2M1 = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64)


def _weight(N, K, g, lo=110, hi=130):
    """Random codes and scale bytes as the library packs them: (QTensor-like codes, scales) in the interchange layout, and the values."""
    code = torch.randint(0, 16, (N, K), generator=g, device="cuda", dtype=torch.uint8)
    scale = torch.randint(lo, hi, (N, K // 32), generator=g, device="cuda", dtype=torch.int64)
    value = E2M1.cuda()[code.long()] * torch.exp2((scale - 127).double()).repeat_interleave(32, 1)
    # interchange: codes [N/32][K/64][32 pairs][32 rows] bytes (low nibble: even k), scales [N/32][K/64][2][32]
    both = (code[:, 0::2] | (code[:, 1::2] << 4)).view(N // 32, 32, K // 64, 32).permute(0, 2, 3, 1).contiguous()
    s = scale.to(torch.uint8).view(N // 32, 32, K // 64, 2).permute(0, 2, 3, 1).contiguous()
    return both, s, value


def _packed(L, parts, N, K):
    import ctypes
    a, b = ctypes.c_size_t(), ctypes.c_size_t()
    pair = len(parts) == 2
    assert L.tpx_tc_packed_bytes(N, K, int(pair), ctypes.byref(a), ctypes.byref(b)) == 0
    wq, sfa = (torch.empty(n.value, device="cuda", dtype=torch.uint8) for n in (a, b))
    p = [t.data_ptr() for part in parts for t in part[:2]] + ([] if pair else [None, None])
    assert L.tpx_repack_mxfp4_tc(*p, N, K, wq.data_ptr(), sfa.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    return wq, sfa


def _check(x, parts, N, K, gamma=None):
    from tpp_pytorch_extension_b200 import _lib
    L, M, pair = _lib.lib(), x.shape[0], len(parts) == 2
    wq, sfa = _packed(L, parts, N, K)
    need = L.tpx_qlinear_mxfp4_tc_scratch_bytes(M, N, K, int(pair))
    sc = torch.zeros(need, device="cuda", dtype=torch.uint8)
    res = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(torch.bfloat16)
    y = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    tail = (M, N, K, None, 2 if pair else 0, None, res.data_ptr(), 0.5, y.data_ptr(), sc.data_ptr(), need, _lib.stream())
    xd = x.double()
    if gamma is None:
        _lib.check(L.tpx_qlinear_mxfp4_tc(wq.data_ptr(), sfa.data_ptr(), int(pair), x.data_ptr(), *tail))
        slack = 0.0
    else:
        _lib.check(L.tpx_rmsnorm_qlinear_mxfp4_tc(wq.data_ptr(), sfa.data_ptr(), int(pair), x.data_ptr(), gamma.data_ptr(), int(gamma.dtype == torch.float32), 1e-5, *tail))
        xd = (xd * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-5) * gamma.double())
        slack = 2.0 ** -8  # the normed value is a bf16 one; the reference's is not rounded
    a, size = xd @ parts[0][2].T, xd.abs() @ parts[0][2].abs().T
    # fp32 sums: a rounding per block of 32 values, group of warps and member, two per product of factors; fp16 activations: 2^-39 of a step's largest
    e = ((K // 32 + 64) * 2.0 ** -24 + slack) * size
    want, err = a, e
    if pair:
        b, size2 = xd @ parts[1][2].T, xd.abs() @ parts[1][2].abs().T
        e2 = ((K // 32 + 64) * 2.0 ** -24 + slack) * size2
        silu = torch.nn.functional.silu(a)
        gate = 1.1 * e + 2.0 ** -18 * silu.abs()  # |silu'| < 1.1; its fast exponential and division
        want, err = silu * b, gate * b.abs() + silu.abs() * e2 + gate * e2
    want = want + 0.5 * res.double()
    bound = 2.0 ** -8 * want.abs() * (1 + 2.0 ** -6) + err * (1 + 2.0 ** -7) + 2.0 ** -22 * res.double().abs()
    assert bool(((y.double() - want).abs() <= bound).all()), float(((y.double() - want).abs() / bound).max())
    return y


# 32 features: a cluster of eight where K allows it; 149 tiles and more: the last CTA has few of its own; 14336: seven tiles per CTA; 16640: no longer one round
@pytest.mark.parametrize("M", [1, 3, 4, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(32, 64), (32, 16448), (1056, 2048), (2400, 192), (4768, 2112), (7136, 320), (9504, 576), (11872, 448), (14336, 704), (16640, 512)])
def test_linear_and_pair(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    parts = [_weight(N, K, g), _weight(N, K, g, 116, 122)]
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    _check(x, parts[:1], N, K)
    small = [(p[0], p[1], p[2]) for p in parts]
    _check((x * 2.0 ** -3).to(torch.bfloat16), small, N, K)
    if K <= 8192:
        gamma = (torch.rand(K, generator=g, device="cuda") + 0.5)
        _check(x, parts[:1], N, K, gamma.to(torch.bfloat16) if M % 2 else gamma)


@pytest.mark.parametrize("M", [2, 8, 12])
def test_activation_sizes(M):
    """Each value's own size from 2^-40 to 2^40, rows of zeros, rows below 2^-120; an infinity stays in its own row."""
    N, K = 160, 1024
    g = torch.Generator(device="cuda").manual_seed(M)
    parts = [_weight(N, K, g)]
    x = torch.randn(M, K, generator=g, device="cuda") * torch.exp2(80 * torch.rand(M, K, generator=g, device="cuda") - 40)
    _check(x.to(torch.bfloat16), parts, N, K)
    x[0] = 0
    x[1] = torch.randn(K, generator=g, device="cuda") * 2.0 ** -120
    y = _check(x.to(torch.bfloat16), parts, N, K)
    x[1, 5] = float("inf")
    z = _check(x.to(torch.bfloat16)[:1], parts, N, K)
    from tpp_pytorch_extension_b200 import _lib
    L = _lib.lib()
    wq, sfa = _packed(L, parts, N, K)
    need = L.tpx_qlinear_mxfp4_tc_scratch_bytes(M, N, K, 0)
    sc, out = torch.zeros(need, device="cuda", dtype=torch.uint8), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    xb = x.to(torch.bfloat16)
    _lib.check(L.tpx_qlinear_mxfp4_tc(wq.data_ptr(), sfa.data_ptr(), 0, xb.data_ptr(), M, N, K, None, 0, None, None, 0.0, out.data_ptr(), sc.data_ptr(), need, _lib.stream()))
    assert bool((~torch.isfinite(out[1])).all()) and bool(torch.isfinite(out[[i for i in range(M) if i != 1]]).all())
    assert z.shape == (1, N) and y.shape == (M, N)


@pytest.mark.parametrize("M", [1, 16])
def test_every_scale_byte(M):
    N, K = 256, 32 * 64
    g = torch.Generator(device="cuda").manual_seed(M)
    for lo, hi, size in ((1, 60, 2.0 ** 60), (60, 190, 1.0), (190, 254, 2.0 ** -80)):
        x = (torch.randn(M, K, generator=g, device="cuda") * size).to(torch.bfloat16)
        parts = [_weight(N, K, g, lo, hi)]
        _check(x, parts, N, K)


@pytest.mark.parametrize("M", [1, 6, 16])
def test_recorded_chain(M):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    from tpp_pytorch_extension_b200.llm.llm_common import quantize_weight
    g = torch.Generator(device="cuda").manual_seed(M)
    w = [quantize_weight((torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).to(torch.bfloat16), "mxfp4")
         for n, k in ((2048, 2048), (4096, 2048), (4096, 2048), (2048, 4096))]
    w[1].prepare(pair_with=w[2])
    gamma = torch.ones(2048, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(M, 2048, generator=g, device="cuda").to(torch.bfloat16)

    def chain(wait):
        y = x
        for _ in range(12):
            o = F.fc_plain_norm(y, gamma, 1e-5, w[0])
            wait()
            h = F.fc_gate_up(o, w[1], w[2])
            wait()
            y = F.fc_plain_act(h, w[3], res=y)
            wait()
        return y

    want = chain(torch.cuda.synchronize)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        chain(lambda: None)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            got = chain(lambda: None)
    for _ in range(3):
        x.copy_(-x)  # other values under way than the run before left
        graph.replay()
        x.copy_(-x)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)


@pytest.mark.parametrize("M", [1, 8])
def test_result_over_activations(M):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    from tpp_pytorch_extension_b200.llm.llm_common import quantize_weight
    g = torch.Generator(device="cuda").manual_seed(M)
    w = quantize_weight((torch.randn(2048, 2048, generator=g, device="cuda") * 0.02).to(torch.bfloat16), "mxfp4")
    x = torch.randn(M, 2048, generator=g, device="cuda").to(torch.bfloat16)
    want = F.fc_plain(x.clone(), w)
    for _ in range(4):
        y = x.clone()
        F.fc_plain(y, w, out=y)
        assert float((y - want).float().norm() / want.float().norm()) < 1e-3  # another group adds the same products


@pytest.mark.parametrize("kind", ["mxfp4", "qint8"])
@pytest.mark.parametrize("M", [1, 2, 8])
def test_norm_weight_of_the_kernel_before(kind, M, monkeypatch):
    """A norm's weight that the kernel in front has just written, into a place that held another."""
    from tpp_pytorch_extension_b200 import _lib
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    from tpp_pytorch_extension_b200.llm.llm_common import quantize_weight
    monkeypatch.setenv("QINT8_BLOCK_SIZE", "64")
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    D = 2048
    w, make = quantize_weight(rnd(D, D) * D ** -0.5, kind), rnd(D, D) * D ** -0.5
    sc = torch.zeros(L.tpx_linear_bf16_tc_scratch_bytes(1, D, D), device="cuda", dtype=torch.uint8)
    x, seeds, gamma = rnd(M, D), rnd(8, 1, D), torch.empty(1, D, device="cuda", dtype=torch.bfloat16)

    def chain(wait):
        ys = []
        for s in seeds:
            _lib.check(L.tpx_linear_bf16_tc(make.data_ptr(), s.data_ptr(), 1, D, D, None, 0, None, None, 0.0, gamma.data_ptr(), sc.data_ptr(), sc.numel(), _lib.stream()))
            wait()
            ys.append(F.fc_plain_norm(x, gamma.view(-1), 1e-5, w))
            wait()
        return torch.stack(ys)

    want = chain(torch.cuda.synchronize)
    assert not torch.equal(want[0], want[1])
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        chain(lambda: None)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            got = chain(lambda: None)
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
