"""32-bit products of very many rows in slabs (csrc/gemm_f32_parts.cu)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_slabs_of_rows():
    """A product whose rows' parts would take more than 256 MB is made in slabs; the scratch does not grow with the rows."""
    from gogguf_b200.csrc import kernels as K
    N, k = 200, 12288
    most = K.f32_parts_scratch(3840, N, k)
    assert all(K.f32_parts_scratch(M, N, k) <= most for M in (1919, 1920, 1921, 2017, 3839, 3841, 100000))
    assert K.f32_parts_scratch(1 << 20, N, k) < 1 << 28
    g = torch.Generator(device="cuda").manual_seed(9)
    w, bias = torch.randn(N, k, device="cuda", generator=g), torch.randn(N, device="cuda", generator=g)
    for M in (1920, 1921, 3900):
        x, out = torch.randn(M, k, device="cuda", generator=g), torch.randn(M, N, device="cuda", generator=g)
        was, scratch = out.clone(), torch.empty(K.f32_parts_scratch(M, N, k), dtype=torch.uint8, device="cuda")
        K.gemm_f32_parts(x, w, out, scratch, accumulate=True, bias=bias)
        want = x.double() @ w.double().T + bias + was
        assert ((out.double() - want).abs() <= (k + 2) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + bias.abs() + was.abs())).all()
