"""The differential attention kernel of any type and size (tpx_diff_attn in fp32, and in bf16 off the tensor-core sizes): token counts around
the four that may share a warp, chunks that end inside such a group, padding, a cache in front, one token. Reference in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# heads, kv_heads, dim, vdim: 16-byte pieces of a key row and not, one to four value columns per lane, wider than four tokens per warp take
HEADS = [(4, 2, 64, 128), (2, 1, 20, 24), (3, 3, 9, 11), (2, 1, 130, 40), (2, 2, 32, 136)]
LAM, MULT, EPS, CAP = 0.3, 0.7, 1e-5, 9.0
# a sum of fp32 products and exponentials, a few 2^-24 each and more where the maps cancel; bf16: the result rounded once, at most 2^-8 of it
TOL = {torch.float32: 2e-5, torch.bfloat16: 2.0 ** -8}


def _want(q, k, v, start, chunk, past):
    """q [B, S, heads, 2, dim], k [B, T, kv, 2, dim], v [B, T, kv, vdim] in float64 -> [B, S, heads, vdim]."""
    B, S, heads = q.shape[:3]
    rep = heads // k.shape[2]
    k, v = k.repeat_interleave(rep, 2), v.repeat_interleave(rep, 2)
    s = CAP * torch.tanh(torch.einsum("bshmd,bthmd->bhmst", q, k) * q.shape[-1] ** -0.5 / CAP)
    at, key = (past + torch.arange(S, device=q.device))[None] - start[:, None], torch.arange(k.shape[1], device=q.device)[None] - start[:, None]
    seen = (key[:, None] >= torch.div(at, chunk, rounding_mode="floor")[:, :, None] * chunk) & (key[:, None] <= at[:, :, None]) & (at[:, :, None] >= 0)
    s = s.masked_fill(~seen[:, None, None], -float("inf"))
    a = torch.nan_to_num(s.softmax(-1))
    o = torch.einsum("bhmst,bthe->bshme", a, v)
    o = o[..., 0, :] - LAM * o[..., 1, :]
    return o / torch.sqrt((o * o).mean(-1, keepdim=True) + EPS) * MULT


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv,dim,vdim", HEADS)
@pytest.mark.parametrize("B,past,S,chunk", [(1, 0, 2, 100), (2, 0, 3, 100), (1, 6, 5, 7), (2, 33, 4, 64), (3, 0, 130, 50), (1, 90, 1, 40), (2, 70, 37, 37),
                                            (40, 0, 97, 33)])
def test_against_64_bits(B, past, S, chunk, heads, kv, dim, vdim, dtype):
    from tpp_pytorch_extension_b200 import _lib
    from tpp_pytorch_extension_b200._C import _hybrid_layers as HL
    g = torch.Generator(device="cuda").manual_seed(B + past + S + dim)
    T, W = past + S, (heads + kv) * 2 * dim + kv * vdim
    proj = torch.randn(B, T, W, generator=g, device="cuda").to(dtype)
    start = torch.tensor([(3 * b) % 8 for b in range(B)], device="cuda", dtype=torch.int32)
    dp = (dim + 15) // 16 * 16
    R, npages = 2 * dp + (vdim + 15) // 16 * 16 + 8, (min(T, chunk) + 31) // 32 + 1
    pages = torch.full((npages, B, kv, 32, R), float("nan"), device="cuda", dtype=dtype)
    table = torch.tensor([p.data_ptr() for p in pages], device="cuda", dtype=torch.int64)

    def call(at, n):
        rows = proj[:, at:at + n].reshape(B * n, W).contiguous()
        out = torch.empty(B * n, heads * vdim, device="cuda", dtype=dtype)
        L = n + (min(at, chunk - 1) if n > 1 else 0)
        live = torch.empty(B, L, kv, R, device="cuda", dtype=dtype)
        HL._call("tpx_diff_attn", _lib.DiffAttnStruct(
            proj=rows.data_ptr(), pages=table.data_ptr(), live=live.data_ptr() if n > 1 else None, start=start.data_ptr(), out=out.data_ptr(), B=B, S=n,
            L=L, past=at, npages=npages, ldp=W, ldo=heads * vdim, heads=heads, kv_heads=kv, dim=dim, vdim=vdim, R=R, chunk=chunk, q_col=0,
            k_col=heads * 2 * dim, v_col=(heads + kv) * 2 * dim, scale=dim ** -0.5, softcap=CAP, lam=LAM, mult=MULT, eps=EPS,
            f32=int(dtype == torch.float32)))
        return out.view(B, n, heads, vdim)

    if past:
        call(0, past)
    got = call(past, S).double()
    p = proj.double()
    want = _want(p[:, past:, :heads * 2 * dim].view(B, S, heads, 2, dim), p[:, :, heads * 2 * dim:(heads + kv) * 2 * dim].view(B, T, kv, 2, dim),
                 p[:, :, (heads + kv) * 2 * dim:].view(B, T, kv, vdim), start.long(), chunk, past)
    assert float((got - want).abs().max()) <= TOL[dtype] * float(want.abs().max())
