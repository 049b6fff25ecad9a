"""Products of 33 to 128 tokens (csrc/gemm_tcgen05.cu): the numbers of tiles, cuts of K and tokens an owner at which the launcher takes another
form, each with a plain output, added into a residual with row statistics, and as a gated unit, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# tokens, tiles of 128 columns, K
FORMS = [
    (33, 8, 1024), (48, 18, 1024), (64, 19, 1024), (40, 32, 1024), (33, 16, 1152),      # one or two slabs a CTA, one CTA an SM or more
    (33, 32, 2048), (48, 32, 2048), (49, 32, 2048), (64, 40, 2048),                     # six or eight warps for an owner's tokens
    (64, 128, 512), (61, 148, 512), (64, 149, 512),                                     # cut in two, not cut
    (33, 149, 3072), (64, 149, 3080), (64, 178, 3080), (47, 222, 3080), (64, 223, 3080),    # two CTAs an SM uncut, three in two cuts
    (64, 296, 256), (33, 297, 256), (64, 444, 256), (64, 445, 256), (50, 592, 256), (64, 593, 256),     # rounds of two and of three an SM
    (65, 32, 2048), (100, 84, 1024), (128, 192, 512),
]


@pytest.mark.parametrize("M,tiles,K_", FORMS)
def test_forms(M, tiles, K_):
    from gogguf_b200.csrc import tcgen05_gemm as T
    g = torch.Generator(device="cuda").manual_seed(M + tiles)
    N = tiles * 128
    x = torch.randn(M, K_, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K_, device="cuda", generator=g) * 0.05).bfloat16()
    want, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # (sums of 16 products at a time, each cut off at 2^-23 of the sum so far, and the adds of up to eight cuts)
    bound = (K_ / 16 + 8) * 2.0 ** -23 * mag
    ragged = torch.full((M, N - 3), -1.0, device="cuda")
    T.gemm_tc(x, w[:N - 3], ragged, cluster=True)
    assert ((ragged.double() - want[:, :N - 3]).abs() <= bound[:, :N - 3]).all()
    res = torch.randn(M, N, device="cuda", generator=g)
    acc, ssq, xhat = res.clone(), torch.empty(M, tiles, device="cuda"), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    norm = torch.rand(M, (K_ + 127) // 128, device="cuda", generator=g) * 128
    f = 1.0 / torch.sqrt(norm.double().sum(1, keepdim=True) / K_ + 1e-6)
    T.gemm_tc_norm(x, w, acc, accumulate=True, in_ssq=norm, eps=1e-6, out_ssq=ssq, out_xhat=xhat)
    new = res.double() + want * f
    assert ((acc.double() - new).abs() <= bound * f + 4 * 2.0 ** -24 * (new.abs() + (want * f).abs())).all()
    assert torch.equal(xhat, acc.bfloat16())
    parts = acc.double().view(M, tiles, 128).square().sum(-1)
    assert ((ssq.double() - parts).abs() <= 128 * 2.0 ** -24 * parts).all()
    act = torch.empty(M, N // 2, device="cuda", dtype=torch.bfloat16)
    T.gemm_tc_norm(x, w, act, swiglu=True, in_ssq=norm, eps=1e-6)
    gate, up = (want * f).view(M, tiles, 2, 64).unbind(2)
    unit = (gate * torch.sigmoid(gate) * up).reshape(M, N // 2)
    off = (bound * f).view(M, tiles, 2, 64).sum(2).reshape(M, N // 2)
    # (an error of either factor times the other, silu's slope at most 1.1, and the rounding to bfloat16)
    room = 1.2 * off * (1 + gate.abs().maximum(up.abs()).reshape(M, N // 2)) + 2.0 ** -8 * unit.abs() + 1e-6
    assert ((act.double() - unit).abs() <= room).all()
