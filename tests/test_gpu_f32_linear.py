"""A 32-bit projection on both sides of the rule that chooses its kernel (parts/base.py, Linear): two layers that share a workspace, numbers
of rows that grow and shrink, with a bias, added into a residual, and rows off 16-byte boundaries."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("fast", [True, False])
def test_two_layers_of_a_workspace(fast):
    from gogguf_b200.csrc import kernels as K
    from gogguf_b200.parts.base import Linear, Runtime, Workspace
    g = torch.Generator(device="cuda").manual_seed(7)
    R = lambda *s: torch.randn(*s, device="cuda", generator=g)                                       # noqa: E731
    rt, ws = Runtime(dtype=torch.float32, device=DEV, fast=fast), Workspace(DEV)
    W, F = 1024, 3072
    up, down = Linear(R(F, W) * 0.03, rt, bias=R(F)), Linear(R(W, F) * 0.02, rt)
    took = set()
    for M in (300, 17, 1, 101, 100, 99, 16, 520, 40, 64, 333, 100):
        took |= {K.f32_parts_pays(M, F, W), K.f32_parts_pays(M, W, F)} if M > 16 else {False}
        for o in (0, 1):
            x, z, res = R(M, W + 4)[:, o:o + W], torch.empty(M, F, device="cuda"), R(M, W)
            was = res.clone()
            up(x, z, ws=ws)
            down(z, res, accumulate=True, ws=ws)
            # (the roundings of a chain of K multiply-adds, and those of the bias and the residual)
            for got, want, mag, k in ((z, x.double() @ up.weight.double().T + up.bias, x.double().abs() @ up.weight.double().abs().T + up.bias.abs(), W),
                                      (res, z.double() @ down.weight.double().T + was, z.double().abs() @ down.weight.double().abs().T + was.abs(), F)):
                assert ((got.double() - want).abs() <= (k + 2) * 2.0 ** -24 * mag).all(), (M, o)
    assert took == {True, False}


def test_the_rule_has_no_step():
    """What is modelled to be the same work within a row does not change its kernel: the rule compares times, it knows no number of rows."""
    from gogguf_b200.csrc import kernels as K
    for N, k in ((512, 512), (1024, 1024), (1024, 3072), (6144, 1024), (2048, 2048), (1800, 4744), (10752, 2048)):
        assert K.f32_parts_pays(99, N, k) == K.f32_parts_pays(100, N, k) == K.f32_parts_pays(101, N, k), (N, k)
        pays = [K.f32_parts_pays(M, N, k) for M in range(64, 640, 64)]           # whole tiles of the CUDA cores
        assert pays == sorted(pays), (N, k, pays)
