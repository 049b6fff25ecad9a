"""CTA-pair products with the tokens as columns (csrc/gemm_tcgen05.cu): numbers of tokens around its tiles, ragged outputs, every output mode, one
and several splits of K, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [129, 160, 161, 290, 333, 384, 566, 576, 577])
@pytest.mark.parametrize("N,K_", [(256, 1024), (2048, 2048), (1000, 520), (331, 2048), (24576, 264)])
def test_modes(M, N, K_):
    from gogguf_b200.csrc import tcgen05_gemm as tc
    g = torch.Generator(device="cuda").manual_seed(M + N)
    need = tc.pair_scratch_elems(M, N, K_)
    scratch = torch.full((max(need, 1),), float("nan"), device="cuda")
    x = torch.randn(M, K_, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K_, device="cuda", generator=g) / math.sqrt(K_)).bfloat16()
    ssq = torch.rand(M, (K_ + 127) // 128, device="cuda", generator=g) * 100 + 60
    prod = x.double() @ w.double().T
    scaled = prod / torch.sqrt(ssq.double().sum(1, keepdim=True) / K_ + 1e-6)
    # (float32 sums of K products, K / 16 truncations of the accumulator)
    bound = 2e-6 + 2e-7 * K_ ** 0.5
    off = lambda a, b: float((a.double() - b).norm() / b.norm())                                       # noqa: E731
    room = torch.full((M + 1, N), -7.0, device="cuda")
    tc.gemm_tc(x, w, room[:M], scratch=scratch, cluster=True)
    assert off(room[:M], prod) < bound and (room[M] == -7.0).all()
    half = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    tc.gemm_tc_norm(x, w, half, in_ssq=ssq, eps=1e-6, scratch=scratch)
    assert off(half, scaled) < 2.0 ** -8
    res = torch.randn(M, N, device="cuda", generator=g)
    acc, xh, oss = res.clone(), torch.empty(M, N, device="cuda", dtype=torch.bfloat16), torch.empty(M, (N + 127) // 128, device="cuda")
    tc.gemm_tc_norm(x, w, acc, accumulate=True, in_ssq=ssq, eps=1e-6, out_ssq=oss, out_xhat=xh, scratch=scratch)
    assert off(acc, res.double() + scaled) < bound and torch.equal(xh, acc.bfloat16())
    parts = torch.nn.functional.pad(acc.double() ** 2, (0, (-N) % 128)).view(M, -1, 128).sum(-1)
    assert off(oss, parts) < 1e-6
    if N % 128 == 0:
        gated = torch.empty(M, N // 2, device="cuda", dtype=torch.bfloat16)
        tc.gemm_tc_norm(x, w, gated, swiglu=True, in_ssq=ssq, eps=1e-6, scratch=scratch)
        blocks = scaled.view(M, N // 128, 2, 64)
        a, b = blocks[:, :, 0].reshape(M, -1), blocks[:, :, 1].reshape(M, -1)
        assert off(gated, a * torch.sigmoid(a) * b) < 2.0 ** -8
    tc.check_status(torch.device("cuda", 0))
