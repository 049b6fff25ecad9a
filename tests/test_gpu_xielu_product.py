"""xIELU in the epilogue of a product (csrc/gemm_tcgen05.cu): every form of the product, ragged sizes, a folded norm, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 16, 17, 61, 128])
@pytest.mark.parametrize("N,K_", [(136, 72), (200, 264), (2048, 1024), (8192, 2048)])
@pytest.mark.parametrize("folded", [False, True])
def test_activation_of_the_sums(M, N, K_, folded):
    from gogguf_b200.csrc import tcgen05_gemm as G
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K_, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K_, device="cuda", generator=g) * 2.0 / K_ ** 0.5).bfloat16()
    ssq = torch.rand(M, (K_ + 127) // 128, device="cuda", generator=g) * 100 + 60 if folded else None
    room = torch.full((M, N + 8), -7.0, device="cuda", dtype=torch.bfloat16)
    G.gemm_tc_xielu(x, w, room[:, :N], 0.9, 1.3, 0.5, in_ssq=ssq, eps=1e-6)
    v = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    if folded:
        f = 1.0 / torch.sqrt(ssq.double().sum(1, keepdim=True) / K_ + 1e-6)
        v, size = v * f, size * f
    act = lambda t: 0.5 * torch.where(t > 0, 0.9 * t * t + 0.5 * t, 1.3 * (torch.expm1(t) - t) + 0.5 * t)     # noqa: E731
    want = act(v)
    # the sums' error (32-bit, cut off) times the largest slope, and the output's rounding to bfloat16
    slope = 0.5 * (1.8 * v.abs() + 2.0)
    assert ((room[:, :N].double() - want).abs() <= want.abs() * 2.0 ** -8 + slope * size * (K_ / 16 + 8) * 2.0 ** -23 + 1e-7).all()
    assert (room[:, N:] == -7.0).all()


def test_more_rows_are_refused():
    from gogguf_b200.csrc import tcgen05_gemm as G
    from gogguf_b200.csrc.build import KernelError
    x, w, out = (torch.zeros(*s, device="cuda", dtype=torch.bfloat16) for s in ((129, 64), (256, 64), (129, 256)))
    with pytest.raises(KernelError):
        G.gemm_tc_xielu(x, w, out, 1.0, 1.0)
