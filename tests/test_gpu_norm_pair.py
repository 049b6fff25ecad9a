"""A norm behind a part, the add into the stream and the norm that comes next in one kernel (csrc/elementwise.cu), against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 8, 511, 512, 700])
@pytest.mark.parametrize("H", [4, 128, 1800, 2048, 4096, 4100, 8192])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rows_of_both_norms(rows, H, dtype):
    from gogguf_b200.csrc import kernels as K
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    x, y = torch.randn(rows, H, device="cuda", generator=g) * 3, torch.randn(rows, H, device="cuda", generator=g)
    w, w2 = torch.rand(H, device="cuda", generator=g) + 0.5, torch.rand(H, device="cuda", generator=g) + 0.5
    out = torch.empty(rows, H, device="cuda", dtype=dtype)
    assert K.rmsnorm_add_norm_takes(x, y, out)
    unit = lambda t, e: t / torch.sqrt((t * t).mean(-1, keepdim=True) + e)                            # noqa: E731
    want = x.double() + unit(y.double(), 1e-6) * w.double()
    then = unit(want, 1e-5) * w2.double()
    K.rmsnorm_add_norm(x, y, w, 1e-6, w2, 1e-5, out, zero_y=True)
    # (sums of H squares in 32 bits: a relative error of a few roundings, as a sum of positive numbers has)
    assert ((x.double() - want).abs() <= 16 * 2.0 ** -24 * (want.abs() + 4)).all() and float(y.abs().max()) == 0.0
    assert ((out.double() - then).abs() <= then.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 0) + 64 * 2.0 ** -24 * (1 + then.abs())).all()


def test_rows_it_does_not_take():
    from gogguf_b200.csrc import kernels as K
    x = torch.zeros(4, 10, device="cuda")
    assert not K.rmsnorm_add_norm_takes(x, x, x)
    with pytest.raises(K.KernelError):
        K.rmsnorm_add_norm(x, x.clone(), x[0], 1e-6, x[0], 1e-6, x.clone())
