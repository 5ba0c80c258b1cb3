"""bf16 linear of few tokens at the edges of its splits: one to twenty tiles per CTA, features and k that end inside a tile, clusters, groups of tokens, padded
leading dimensions; and a recorded chain of calls. Reference: 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 16 and 100 features: clusters; 2390 and more: 150, 300, ... tiles, the last CTA with few of its own; 47200: twenty per CTA
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(16, 8), (100, 4104), (2390, 200), (4768, 72), (7130, 328), (9504, 136), (11872, 64), (14240, 192), (18950, 248), (28400, 128), (47200, 40)])
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
    out = HL.linear(x, wide[:, :K], out_f32=True) if wide.stride(0) % 8 == 0 else HL.linear(x, w, out_f32=True)
    assert bool(((out.double() - sums).abs() <= err + 2.0 ** -23 * size).all())


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
