"""int8 linear of few tokens at the edges of its splits: tiles per CTA, the last CTA's overlap, clusters, odd and missing k blocks, groups of
tokens; the gate/up pair; and a recorded chain of calls, in which every kernel starts before the one in front of it has ended. Reference: the
same arithmetic in 64 bits."""
import pytest
import torch

from tests.test_gpu_int8_steps import _reference

pytestmark = pytest.mark.gpu


def _weight(N, K, g):
    Np, Kp = (N + 127) // 128 * 128, (K + 127) // 128 * 128
    q = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    s = torch.rand(K // 64, N, generator=g, device="cuda") * 0.01
    wq = torch.zeros(Np, Kp, device="cuda", dtype=torch.int8)
    sw = torch.zeros(K // 64, Np, device="cuda")
    wq[:N, :K], sw[:, :N] = q, s
    return q, s, wq, sw


# 16 features: a cluster of eight where K allows it; 149, 297, ... tiles: the last CTA has one of its own; 1037 and 1193 tiles: two rounds; the last five
# as long as five, six and seven tiles per CTA and two rounds have to be for more than 8 and 16 tokens
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(16, 64), (16, 16448), (1040, 1024), (2384, 192), (4752, 2112), (7120, 320), (9488, 576), (11856, 448), (14224, 704), (16592, 1024), (9488, 1600),
                                 (11856, 3136), (14224, 4160), (19088, 320), (19088, 1600)])
def test_linear_and_pair(M, N, K):
    from tpp_pytorch_extension_b200 import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    q, s, wq, sw = _weight(N, K, g)
    q2, s2, wq2, sw2 = _weight(N, K, g)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    res = torch.randn(M, N, generator=g, device="cuda").to(torch.bfloat16)
    need = L.tpx_qlinear_qint8_tc_scratch_bytes(M, N, K, 64)
    sc = torch.zeros(need, device="cuda", dtype=torch.uint8)
    y, h = (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in "yh")
    _lib.check(L.tpx_qlinear_qint8_tc(wq.data_ptr(), sw.data_ptr(), x.data_ptr(), None, 0, 0.0, M, N, K, 64, 0, None, 0, None, res.data_ptr(), 0.5,
                                      y.data_ptr(), sc.data_ptr(), need, _lib.stream()))
    _lib.check(L.tpx_qlinear_qint8_pair_tc(wq.data_ptr(), sw.data_ptr(), wq2.data_ptr(), sw2.data_ptr(), x.data_ptr(), None, 0, 0.0, M, N, K, 64, 2,
                                           h.data_ptr(), sc.data_ptr(), need, _lib.stream()))
    a, size = _reference(x, q, s, 64)
    b, size2 = _reference(x, q2, s2, 64)
    # a block's term is rounded three times in 32 bits, sums once per block and part; the result once to bf16 (half a unit: 2^-8 of it at most)
    e1, e2 = ((K // 64 + 40) * 2.0 ** -24 * z for z in (size, size2))
    want = a + 0.5 * res.double()
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() * (1 + 2.0 ** -10) + e1 + 2.0 ** -23 * (size + res.double().abs())).all())
    # |silu'| < 1.1; its fast exponential and division: 2^-18 of the value. Above 16 tokens the gate is a bf16 value before it meets the other sum.
    silu = torch.nn.functional.silu(a)
    want = silu * b
    gate = 1.1 * e1 + (2.0 ** -18 + (2.0 ** -8 if M > 16 else 0)) * silu.abs()
    bound = 2.0 ** -8 * want.abs() * (1 + 2.0 ** -6) + (gate * b.abs() + silu.abs() * e2 + gate * e2) * (1 + 2.0 ** -7)
    assert bool(((h.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("M", [1, 16, 32])
def test_recorded_chain(M, monkeypatch):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    from tpp_pytorch_extension_b200.llm.llm_common import quantize_weight
    monkeypatch.setenv("QINT8_BLOCK_SIZE", "64")
    g = torch.Generator(device="cuda").manual_seed(M)
    w = [quantize_weight((torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).to(torch.bfloat16), "qint8")
         for n, k in ((2048, 2048), (4096, 2048), (4096, 2048), (2048, 4096))]
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


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("K,f32", [(64, False), (4096, True), (4160, False), (8192, True), (8192, False)])
def test_norm_and_reuse(M, K, f32):
    from tpp_pytorch_extension_b200 import _lib
    L, N = _lib.lib(), 272
    g = torch.Generator(device="cuda").manual_seed(M + K)
    q, s, wq, sw = _weight(N, K, g)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    gamma = torch.randn(K, generator=g, device="cuda").to(torch.float32 if f32 else torch.bfloat16)
    need = L.tpx_qlinear_qint8_tc_scratch_bytes(M, N, K, 64)
    sc = torch.zeros(need, device="cuda", dtype=torch.uint8)
    y, again = (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in "ya")

    def call(x, gamma, reuse, y):
        _lib.check(L.tpx_qlinear_qint8_tc(wq.data_ptr(), sw.data_ptr(), x.data_ptr(), _lib.ptr(gamma), int(f32), 1e-5, M, N, K, 64, reuse, None, 0, None, None, 0.0,
                                          y.data_ptr(), sc.data_ptr(), need, _lib.stream()))

    call(x, gamma, 0, y)
    call(torch.zeros_like(x), None, 1, again)  # what the call before left in the scratch
    assert torch.equal(y, again)
    normed = (x.double() * (x.double().square().mean(-1, keepdim=True) + 1e-5).rsqrt() * gamma.double()).to(torch.bfloat16)
    a, _ = _reference(normed, q, s, 64)
    # a normed value may round to the neighbouring bf16 and its int8 to the neighbouring step: one step in a few of K values, random signs
    assert float((y.double() - a).norm() / a.norm()) < 2.0 ** -8


@pytest.mark.parametrize("M", [1, 2])
def test_result_over_activations(M, monkeypatch):
    from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
    from tpp_pytorch_extension_b200.llm.llm_common import quantize_weight
    monkeypatch.setenv("QINT8_BLOCK_SIZE", "64")
    g = torch.Generator(device="cuda").manual_seed(M)
    w = quantize_weight((torch.randn(2048, 2048, generator=g, device="cuda") * 0.02).to(torch.bfloat16), "qint8")
    x = torch.randn(M, 2048, generator=g, device="cuda").to(torch.bfloat16)
    want = F.fc_plain(x.clone(), w)
    for _ in range(4):
        y = x.clone()
        F.fc_plain(y, w, out=y)
        assert torch.equal(y, want)


# 272, 14224 and 17408 features: 17, 889 and 1088 tiles of 16, which different kernels take above 8, 16 and 2 tokens; 320: half a step of 128 k values left over
@pytest.mark.parametrize("M", [1, 2, 8, 16, 17, 24, 32, 33])
@pytest.mark.parametrize("first,second", [(272, 14224), (14224, 272), (272, 17408), (17408, 272), (272, 272)])
@pytest.mark.parametrize("K", [320, 4096])
def test_reuse_across_sizes(M, first, second, K):
    from tpp_pytorch_extension_b200 import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(M + first)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    gamma = torch.randn(K, generator=g, device="cuda")
    need = max(L.tpx_qlinear_qint8_tc_scratch_bytes(M, N, K, 64) for N in (first, second))
    sc = torch.zeros(need, device="cuda", dtype=torch.uint8)

    def call(w, x, gamma, reuse):
        y = torch.empty(M, w[0].shape[0], device="cuda", dtype=torch.bfloat16)
        _lib.check(L.tpx_qlinear_qint8_tc(w[2].data_ptr(), w[3].data_ptr(), x.data_ptr(), _lib.ptr(gamma), 1, 1e-5, M, y.shape[1], K, 64, reuse, None, 0, None, None, 0.0,
                                          y.data_ptr(), sc.data_ptr(), need, _lib.stream()))
        return y

    a, b = _weight(first, K, g), _weight(second, K, g)
    want = call(b, x, gamma, 0)
    call(a, x, gamma, 0)
    assert torch.equal(call(b, torch.zeros_like(x), None, 1), want)  # what the call before left in the scratch
