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


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_weights_that_are_views_of_a_packed_tensor(tmp_path, dtype):
    """A float32 norm weight is kept where the caller has it, which may be off a 16-byte boundary: the same model either way."""
    from gogguf_b200.config import config_from_dict
    from gogguf_b200.engine import Model, StepEntry, Stepper
    from helpers import random_tokens, read_folder
    from sokirax_cases import make_folder
    cfg, w = read_folder(make_folder(tmp_path, "S", "float32"))
    assert cfg["width"] % 4 == 0
    w = {n: t.to("cuda", getattr(torch, dtype) if t.dim() > 1 else torch.float32) for n, t in w.items()}
    vectors = [n for n, t in w.items() if t.dim() == 1]
    packed, at, views = torch.empty(sum(w[n].numel() + 4 for n in vectors) + 1, device="cuda"), 1, dict(w)
    for n in vectors:
        views[n] = packed[at:at + w[n].numel()].copy_(w[n])
        at += -(-w[n].numel() // 4) * 4              # (every one of them a float behind a boundary)
        assert views[n].data_ptr() % 16 == 4
    out = []
    for weights in (w, views):
        model = Model(config_from_dict(cfg).to_spec(), dict(weights), dtype=dtype)
        cache = model.new_cache(max_tokens=256)
        st, slot = Stepper(model, cache), cache.open()
        tokens = random_tokens(cfg["vocab"], 21, 3)
        out.append([st.step([StepEntry(slot, tokens[:20], want=[19])]).clone(), st.step([StepEntry(slot, tokens[20:], want=[0])]).clone()])
    for a, b in zip(*out):                           # (other orders of the norms' sums)
        assert (a - b).norm() <= (1e-5 if dtype == "float32" else 2e-2) * a.norm()
