"""bf16 linear of few tokens at the edges of its splits: one to twenty tiles per CTA, features and k that end inside a tile, clusters, groups of tokens, padded
leading dimensions, every epilogue; a recorded chain of calls; a result over its own activations. Reference: 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 16 and 100 features: clusters; 2390 and more: 150, 300, ... tiles, the last CTA with few of its own; 47200: twenty per CTA; 1032 values: as long
# as five to eight tiles per CTA have to be above 16 tokens
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(16, 8), (100, 4104), (2390, 200), (4768, 72), (7130, 328), (9504, 136), (11872, 64), (14240, 192), (18950, 248), (28400, 128), (47200, 40),
                                 (9500, 1032), (11872, 1032), (14240, 1032), (17000, 1032)])
def test_plain_and_strided(M, N, K):
    from tpp_pytorch_extension_b200 import _lib
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    from tpp_pytorch_extension_b200._C import _hybrid_layers as HL
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    wide = torch.randn(N, K + 24, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)
    mul, res = (torch.randn(M, N, generator=g, device="cuda").to(torch.bfloat16) for _ in "ab")
    w = wide[:, :K].contiguous()
    y = F.fc_plain_act(x, w, bias, "relu", mul_in=mul, res=res, res_scale=0.5)
    sums, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    err = (K // 16 + 40) * 2.0 ** -23 * (size + bias.double().abs())  # an MMA's sum of sixteen products is cut off at 32 bits, a group's added rounded
    want = (sums + bias.double()).clamp(min=0) * mul.double() + 0.5 * res.double()
    bound = 2.0 ** -8 * want.abs() * (1 + 2.0 ** -6) + err * mul.double().abs() + 2.0 ** -22 * (size * mul.double().abs() + res.double().abs())
    assert bool(((y.double() - want).abs() <= bound).all())
    # rows of a wider matrix, fp32 result
    out = HL.linear(x, wide[:, :K], out_f32=True)
    assert bool(((out.double() - sums).abs() <= err + 2.0 ** -23 * size).all())


# 96 features of 4104 values: a cluster cuts k; 2390: the last CTA has few of its own, and the gated units start inside a CTA's tiles
@pytest.mark.parametrize("M", [1, 8, 9, 17, 32])
@pytest.mark.parametrize("N,K,act_from", [(96, 4104, 0), (98, 4104, 42), (2390, 200, 1002), (4768, 72, 4766), (7130, 328, 7130), (28400, 128, 10000)])
def test_gated_units(M, N, K, act_from):
    from tpp_pytorch_extension_b200._C import _hybrid_layers as HL
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, bias, limit = rnd(M, K).to(torch.bfloat16), (rnd(N, K) * 3 * K ** -0.5).to(torch.bfloat16), rnd(N), 2.5
    units = (N - act_from) // 2
    z = torch.full((M, units + 3), 7.0, device="cuda", dtype=torch.bfloat16)
    y = HL.linear_glu(x, w, bias, act_from, limit, z)
    v, err = x.double() @ w.double().T + bias.double(), (K // 16 + 40) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T + bias.double().abs())
    assert bool(((y.double() - v[:, :act_from]).abs() <= 2.0 ** -8 * v[:, :act_from].abs() + err[:, :act_from] * 2).all())
    a, b, ea, eb = v[:, act_from::2], v[:, act_from + 1::2], err[:, act_from::2], err[:, act_from + 1::2]
    gate, up = a.clamp(max=limit), b.clamp(-limit, limit) + 1
    act = gate * torch.sigmoid(1.702 * gate)  # its slope is below 1.1; fast exponential and division, 2^-18 of the value
    want = act * up
    bound = 2.0 ** -8 * want.abs() * (1 + 2.0 ** -6) + (1.1 * ea + 2.0 ** -18 * act.abs()) * up.abs() + (act.abs() + 1.1 * ea) * eb
    assert bool(((z[:, :units].double() - want).abs() <= bound).all())
    assert bool((z[:, units:] == 7).all())


@pytest.mark.parametrize("M", [1, 8, 9, 17, 32])
@pytest.mark.parametrize("N,K", [(96, 4104), (100, 4104), (2390, 200), (4768, 72), (28400, 128)])
@pytest.mark.parametrize("extra", [False, True])
def test_residual_and_norm(M, N, K, extra):
    from tpp_pytorch_extension_b200._C import _hybrid_layers as HL
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w = rnd(M, K).to(torch.bfloat16), (rnd(N, K) * K ** -0.5).to(torch.bfloat16)
    res, add, nw, nb, alpha = rnd(M, N), rnd(N) if extra else None, rnd(N), rnd(N), 0.7
    s, h = HL.linear_residual(x, w, res, add, (alpha, nw, nb))
    v = x.double() @ w.double().T
    want = res.double() + v + (add.double() if extra else 0)
    err = (K // 16 + 40) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T) + 2.0 ** -23 * (res.double().abs() + v.abs() + (add.double().abs() if extra else 0))
    assert bool(((s.double() - want).abs() <= err).all())
    t = torch.tanh(alpha * want)
    want = t * nw.double() + nb.double()
    # tanh to 2^-21, its slope at most 1, the product and sum rounded once
    bound = 2.0 ** -8 * want.abs() * (1 + 2.0 ** -6) + (alpha * err + 2.0 ** -21) * nw.double().abs() + 2.0 ** -23 * want.abs()
    assert bool(((h.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("M", [1, 16, 24])
def test_recorded_chain(M):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    g = torch.Generator(device="cuda").manual_seed(M)
    w = [(torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).to(torch.bfloat16) for n, k in ((2048, 2048), (4096, 2048), (2048, 4096))]
    x = torch.randn(M, 2048, generator=g, device="cuda").to(torch.bfloat16)

    def chain(wait):
        y = x
        for _ in range(12):
            o = F.fc_plain(y, w[0])
            wait()
            h = F.fc_plain_act(o, w[1], None, "silu")
            wait()
            y = F.fc_plain_act(h, w[2], res=y)
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


@pytest.mark.parametrize("M", [1, 8, 17, 32])
@pytest.mark.parametrize("N,K", [(16, 16), (128, 128), (128, 4096), (120, 200)])
def test_result_over_activations(M, N, K):
    """Up to 128 features: into the activations' own memory, from its start, from its end, with and without the activations' row stride."""
    from tpp_pytorch_extension_b200 import _lib
    from tpp_pytorch_extension_b200._C import _hybrid_layers as HL
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    sc = torch.zeros(L.tpx_linear_bf16_tc_scratch_bytes(M, N, K), device="cuda", dtype=torch.uint8)
    want = x.double() @ w.double().T
    err = (K // 16 + 40) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    for _ in range(4):
        for at in (0, M * K - M * N):
            if at < 0:
                continue
            buf = x.clone().flatten()
            y = buf[at:at + M * N].view(M, N)
            _lib.check(L.tpx_linear_bf16_tc(w.data_ptr(), buf.data_ptr(), M, N, K, None, 0, None, None, 0.0, y.data_ptr(), sc.data_ptr(), sc.numel(), _lib.stream()))
            assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + err).all())
        buf = torch.empty(M, K + 8, device="cuda", dtype=torch.bfloat16)
        buf[:, :K] = x
        y = buf[:, K - min(N, K):K - min(N, K) + N]
        HL._linear_call(buf[:, :K], w, y)
        assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + err).all())
