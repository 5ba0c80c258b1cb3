"""int8 linear at the edges of its steps: every token tile and block size, a CTA per tile and clusters that cut K, k padding, odd groups of
steps, the largest block sums. Reference: the same arithmetic (activations quantised per block, whole-number block products) in 64 bits."""
import pytest
import torch

from tests.gpu_util import assert_no_kernel_error

pytestmark = pytest.mark.gpu

def _reference(x, q, s, block):
    M, K = x.shape
    xb = x.float().view(M, -1, block)
    sx = (xb.abs().amax(-1).double() / 127.0).float()
    inv = torch.where(sx != 0, 1.0 / sx, torch.zeros_like(sx))
    xq = torch.round(xb * inv.unsqueeze(-1)).clamp(-127, 127).double()
    wq = q.double().view(q.shape[0], -1, block)
    y = torch.zeros(M, q.shape[0], dtype=torch.float64, device=x.device)
    size = torch.zeros_like(y)  # of all terms of a sum
    for b in range(K // block):
        t = (xq[:, b] @ wq[:, b].T) * sx[:, b:b + 1].double() * s[b].double()
        y += t
        size += t.abs()
    return y, size


@pytest.mark.parametrize("M", [1, 17, 64, 128, 200])
@pytest.mark.parametrize("N,K,block", [(11008, 1088, 64), (4096, 2048, 64), (6144, 1152, 128), (2064, 2048, 256), (512, 2560, 512), (9600, 576, 64), (128, 64, 64)])
def test_against_the_same_arithmetic(M, N, K, block):
    from tpp_pytorch_extension_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    Np, Kp = (N + 127) // 128 * 128, (K + 127) // 128 * 128
    q = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    q[3], q[5] = 127, -127  # the largest sums
    wq = torch.zeros(Np, Kp, device="cuda", dtype=torch.int8)
    wq[:N, :K] = q
    s = torch.rand(K // block, N, generator=g, device="cuda") * 0.01
    sw = torch.zeros(K // block, Np, device="cuda")
    sw[:, :N] = s
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    x[0] = 2.0
    bias = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)
    y = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    L = _lib.lib()
    need = L.tpx_qlinear_qint8_tc_scratch_bytes(M, N, K, block)
    sc = torch.zeros(need, device="cuda", dtype=torch.uint8)
    want, size = _reference(x, q, s, block)
    want, size = want + bias.double(), size + bias.double().abs()
    _lib.check(L.tpx_qlinear_qint8_tc(wq.data_ptr(), sw.data_ptr(), x.data_ptr(), None, 0, 0.0, M, N, K, block, 0, bias.data_ptr(), 0, None, None,
                                      1.0, y.data_ptr(), sc.data_ptr(), need, _lib.stream()))
    # element by element: half a unit of a bf16 result is at most 2^-8 of it; a block's term is rounded three times in 32 bits (whole number times
    # scale, times scale, sum; the sum's part at most (blocks + 1) 2^-24 of all terms), and so are parts of a cluster
    bound = 2.0 ** -8 * want.abs() * (1 + 2.0 ** -10) + (K // block + 12) * 2.0 ** -24 * size
    assert bool(((y.double() - want).abs() <= bound).all())
    assert int(sc[65532:65536].view(torch.int32)) == 0
    assert_no_kernel_error()
