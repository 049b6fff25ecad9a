"""The products refuse an output that has no room for their rows, whatever its shape says: the launchers get a pointer and a
row stride and cannot see where the tensor ends.  Launchers are replaced, so nothing runs on a device."""
import pytest
import torch

from gogguf_b200.csrc import kernels, tcgen05_gemm
from gogguf_b200.csrc.build import KernelError

M, N, K = 3, 128, 64


@pytest.fixture
def launched(monkeypatch):
    calls = []
    for mod in (kernels, tcgen05_gemm):
        monkeypatch.setattr(mod, "kernel", lambda module, name: lambda *args: calls.append(name))
        monkeypatch.setattr(mod, "stream_ptr", lambda: 0)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    monkeypatch.setattr(kernels, "_p", lambda t: 0 if t is None else t.data_ptr())
    monkeypatch.setattr(tcgen05_gemm, "status_word", lambda device: torch.zeros(1, dtype=torch.int32))
    return calls


def bf(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16)


FORMS = {
    "plain": lambda x, out, m: kernels.gemm_plain(x, bf(N, K), out, m=m),
    "tc": lambda x, out, m: tcgen05_gemm.gemm_tc(x, bf(N, K), out, m=m),
    "norm": lambda x, out, m: tcgen05_gemm.gemm_tc_norm(x, bf(N, K), out, m=m, in_ssq=torch.zeros(16, 1)),
    "gated": lambda x, out, m: tcgen05_gemm.gemm_tc(x, bf(2 * N, K), out, m=m, swiglu=True),
    "gated norm": lambda x, out, m: tcgen05_gemm.gemm_tc_norm(x, bf(2 * N, K), out, m=m, swiglu=True, in_ssq=torch.zeros(16, 1)),
}


@pytest.mark.parametrize("form", FORMS)
def test_outputs_without_room_are_refused(form, launched):
    wide = bf(8, 2 * N)
    for out, m in ((bf(1, M, N), M),                 # logits.unsqueeze_(0): the stride between "rows" is the whole tensor
                   (bf(M, N), M + 1),                # fewer rows than the product writes
                   (bf(2, M, N), 2 * M),
                   (wide[5:, :N], M + 1), (wide[::4, N:], M)):
        with pytest.raises(KernelError):
            FORMS[form](bf(8, K), out, m)
    assert launched == []


@pytest.mark.parametrize("form", FORMS)
def test_outputs_with_room_are_taken(form, launched):
    wide = bf(8, 2 * N)
    good = [(bf(M, N), M), (bf(8, N), M), (bf(1, 1, N), 1), (bf(M, 1, N), M), (wide[5:, :N], M), (wide[5:, N:], M), (wide[::3, N:], M),
            (bf(0, N), 0)]
    for out, m in good:
        FORMS[form](bf(8, K), out, m)
    assert len(launched) == len(good)
