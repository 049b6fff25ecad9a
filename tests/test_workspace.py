"""Scratch buffers hand out a tensor of the caller's own each time: what a caller or a registered part does in place to the
shape, the strides or the flags of one stays with that one (the products take a row's stride from the tensor they get)."""
from types import SimpleNamespace

import pytest
import torch

from gogguf_b200.parts.base import Workspace

IN_PLACE = {
    "unsqueeze_": lambda t: t.unsqueeze_(0),
    "squeeze_": lambda t: t.squeeze_(),
    "t_": lambda t: t.t_(),
    "resize_": lambda t: t.resize_(1, t.numel()),
    "requires_grad_": lambda t: t.requires_grad_(),
}


def layout(t):
    return tuple(t.shape), t.stride(), t.storage_offset(), t.requires_grad


@pytest.mark.parametrize("change", IN_PLACE, ids=list(IN_PLACE))
@pytest.mark.parametrize("rows", [1, 3])
def test_a_changed_view_is_the_callers_own(change, rows):
    ws = Workspace(torch.device("cpu"))
    first = ws.get("logits", (rows, 64), torch.float32)
    want, address = layout(first), first.data_ptr()
    IN_PLACE[change](first)
    again = ws.get("logits", (rows, 64), torch.float32)
    assert layout(again) == want and again.data_ptr() == address


def test_views_follow_their_buffer():
    ws = Workspace(torch.device("cpu"))
    small = ws.get("x", (2, 3), torch.float32)
    small.fill_(1.0)
    assert torch.equal(ws.get("x", (6,), torch.float32), torch.ones(6))          # one buffer behind every shape
    big = ws.get("x", (5, 3), torch.float32)
    assert ws.get("x", (2, 3), torch.float32).data_ptr() == big.data_ptr()      # no view of the buffer that was too small
    for n in range(Workspace.MAX_VIEWS + 10):
        assert tuple(ws.get("x", (1, n % 15 + 1), torch.float32).shape) == (1, n % 15 + 1)


@pytest.mark.parametrize("change", IN_PLACE, ids=list(IN_PLACE))
@pytest.mark.parametrize("rows", [1, 3])
def test_head_after_changed_logits(change, rows):
    """The row stride that the head's product is given does not depend on what was done to the logits before."""
    from gogguf_b200.engine.step import Stepper
    given = []
    model = SimpleNamespace(rt=SimpleNamespace(device=torch.device("cpu"), dtype=torch.float32),
                            spec=SimpleNamespace(hidden_size=8, vocab_size=64),
                            final_norm=SimpleNamespace(forward=lambda x, out, r: given.append(layout(out))),
                            head=SimpleNamespace(forward=lambda h, out, ctx, m: given.append(layout(out))))
    stepper = Stepper(model, None)
    ctx = SimpleNamespace(ws=stepper.ws)
    x, wanted = torch.zeros(rows, 8), torch.arange(rows, dtype=torch.int32)
    for _ in range(2):
        logits = stepper.run_head(ctx, x, wanted, rows)
        assert tuple(logits.shape) == (rows, 64) and logits.stride() == (64, 1)
        IN_PLACE[change](logits)
    assert given[:2] == given[2:]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_steps_after_changed_logits(dtype, tmp_path):
    """Eager steps of one size after the logits of the last were reshaped in place: the same shape and values."""
    import gogguf_b200 as gg
    from helpers import make_folder
    ctx = gg.load(make_folder(tmp_path, "L", dtype), gg.LoadOptions(dtype=dtype, max_tokens=512)).new_context()
    for want in ([4], [0, 2, 4]):
        first = None
        for change in [None] + list(IN_PLACE):
            slot = ctx.cache.open()
            logits = ctx.stepper.step([gg.StepEntry(slot, [5, 7, 9, 11, 13], want=want)])
            assert tuple(logits.shape) == (len(want), 1000) and logits.stride() == (1000, 1) and not logits.requires_grad
            first = logits.clone() if first is None else first
            assert torch.equal(logits, first)
            ctx.cache.close(slot)
            if change is not None:
                IN_PLACE[change](logits)
