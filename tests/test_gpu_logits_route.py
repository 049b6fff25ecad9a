"""Router logits and the choice in one kernel (csrc/moe.cu): the bits of the two kernels it stands for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,W,E,top", [(1, 4, 1, 1), (8, 2048, 16, 2), (148, 1024, 32, 8), (5, 100, 7, 7), (3, 1028, 31, 4), (2, 12000, 9, 2)])
@pytest.mark.parametrize("softmax,renorm,real,scale", [(False, False, 0, 1.0), (True, True, 0, 2.5), (True, False, 1, 1.0)])
@pytest.mark.parametrize("dtypes", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32)])
def test_same_bits(T, W, E, top, softmax, renorm, real, scale, dtypes):
    from gogguf_b200.csrc import kernels as K
    g = torch.Generator(device="cuda").manual_seed(T + W)
    h, wr = torch.randn(T, W, device="cuda", generator=g).to(dtypes[0]), torch.randn(E, W, device="cuda", generator=g).to(dtypes[1])
    if E > 2:
        wr[E - 1] = wr[0]                                # equal logits: the lower expert comes first
    seq = torch.arange(T, device="cuda", dtype=torch.int32)
    if T > 2:
        seq[1] = -1
    outs = []
    for fused in (False, True):
        z, idx, wts = torch.empty(T, E, device="cuda"), torch.full((T, top), -9, device="cuda", dtype=torch.int32), torch.empty(T, top, device="cuda")
        if fused:
            assert K.moe_logits_route_takes(h, wr, T)
            K.moe_logits_route(h, wr, z, top, idx, wts, seq, T, softmax=softmax, renormalize=renorm, n_real=real, scale=scale)
        else:
            K.moe_router_logits(h, wr, z, T)
            K.moe_route(z, top, idx, wts, seq, softmax=softmax, renormalize=renorm, rows=T, n_real=real, scale=scale)
        outs.append((z, idx, wts))
    assert all(torch.equal(a, b) for a, b in zip(*outs))


def test_what_it_leaves_to_the_two():
    from gogguf_b200.csrc import kernels as K
    x = lambda *s: torch.zeros(*s, device="cuda")                                                     # noqa: E731
    assert not K.moe_logits_route_takes(x(149, 8), x(4, 8), 149) and not K.moe_logits_route_takes(x(2, 8), x(33, 8), 2)
    assert not K.moe_logits_route_takes(x(2, 6), x(4, 6), 2) and not K.moe_logits_route_takes(x(2, 12004), x(4, 12004), 2)
