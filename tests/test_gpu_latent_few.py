"""Per-head products of few tokens and the merge of the attention's shares inside them (csrc/latent_attention.cu), against float64 and
against the two kernels they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 5, 16, 17])
@pytest.mark.parametrize("N,K_", [(64, 256), (256, 64), (30, 8), (100, 200), (65, 40), (64, 264)])
@pytest.mark.parametrize("gated", [False, True])
def test_products_of_few_tokens(M, N, K_, gated):
    from gogguf_b200.csrc import fast_latent
    g = torch.Generator(device="cuda").manual_seed(M + N)
    H = 3
    x = torch.randn(M, H * (K_ + 8), device="cuda", generator=g).bfloat16()
    w = torch.randn(H, N, K_, device="cuda", generator=g).bfloat16()
    gate = torch.randn(M, H * N, device="cuda", generator=g) if gated else None
    out = torch.full((M, H, N + 2), -7.0, device="cuda")
    fast_latent.headwise_gemm_mma(x, x.stride(0), K_ + 8, w, out, H * (N + 2), N + 2, M, 0.5, gate)
    want = 0.5 * torch.einsum("mhk,hnk->mhn", x.view(M, H, -1)[..., :K_].double(), w.double())
    if gated:
        want = want * torch.sigmoid(gate.double()).view(M, H, N)
    size = torch.einsum("mhk,hnk->mhn", x.view(M, H, -1)[..., :K_].double().abs(), w.double().abs())
    # (products of bfloat16 are exact in 32 bits; K sums, cut off at worst, and a few roundings of the gate)
    assert ((out[..., :N].double() - want).abs() <= size * (K_ + 8) * 2.0 ** -23).all()
    assert (out[..., N:] == -7.0).all()


@pytest.mark.parametrize("M,H,R,N,splits", [(1, 16, 256, 64, 32), (4, 16, 256, 64, 14), (16, 3, 64, 100, 2), (5, 2, 136, 30, 9)])
@pytest.mark.parametrize("sunk", [False, True])
def test_merge_of_shares(M, H, R, N, splits, sunk):
    from gogguf_b200.csrc import fast_latent
    g = torch.Generator(device="cuda").manual_seed(M * R)
    part_o = torch.randn(M * H, splits, R, device="cuda", generator=g)
    ml = torch.stack([torch.randn(M * H, splits, device="cuda", generator=g) * 4, torch.rand(M * H, splits, device="cuda", generator=g) + 1.0], -1)
    empty = torch.rand(M * H, splits, device="cuda", generator=g) < 0.3
    empty[:, 0] = False
    ml[empty] = torch.tensor([-float("inf"), 0.0], device="cuda")
    part_o[empty] = 0.0
    uv = torch.randn(H, N, R, device="cuda", generator=g).bfloat16()
    sink = torch.randn(H, device="cuda", generator=g) if sunk else None
    seq = torch.arange(M, device="cuda", dtype=torch.int32)
    if M > 2:
        seq[1] = -1                                       # a row of padding
    out = torch.empty(M, H * N, device="cuda", dtype=torch.bfloat16)
    fast_latent.expand_shares(part_o, ml.contiguous(), seq, uv, out, M, 0.5, sink=sink)
    m, l, o = ml[..., 0].double(), ml[..., 1].double(), part_o.double()
    top = m.amax(1)
    if sunk:
        sk = (sink.double() * 1.4426950408889634).repeat(M)
        top = torch.maximum(top, sk)
    f = torch.exp2(m - top[:, None])
    L = (f * l).sum(1) + (torch.exp2(sk - top) if sunk else 0.0)
    lat = ((f[..., None] * o).sum(1) / L[:, None]).float().bfloat16().double().view(M, H, R)
    want = 0.5 * torch.einsum("mhr,hnr->mhn", lat, uv.double())
    want[seq < 0] = 0.0
    # (the latent's rounding to bfloat16 may fall to the other side, and the output is rounded to bfloat16)
    size = 0.5 * torch.einsum("mhr,hnr->mhn", lat.abs(), uv.double().abs())
    assert ((out.view(M, H, N).double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -8 * 0.25 + 1e-6).all()
    assert M <= 2 or (out[1] == 0).all()
