"""Which form a step's routed experts take (parts/experts.py): the launchers are replaced by names, nothing runs on a device."""
from types import SimpleNamespace

import pytest
import torch

from gogguf_b200.parts import experts
from gogguf_b200.parts.base import Workspace


def route(monkeypatch, E, W, F, top, T, decode=False):
    calls = []
    for name in ("moe_place_gather", "moe_grouped", "moe_combine", "moe_gather", "moe_expert_mma", "moe_gate_up", "moe_down"):
        monkeypatch.setattr(experts.K, name, lambda *a, _n=name, **k: calls.append(_n))
    part = experts.RoutedExperts.__new__(experts.RoutedExperts)
    part.E, part.R, part.hidden, part.inter, part.top = E, E, W, F, top
    part.identity, part.on_input, part._mma = 0, False, True
    part.limit, part.slope, part.up_offset, part.out_scale = 1.0, 1.0, 0.0, 1.0
    part.w_gu = part.w_d = None
    part.route = lambda h, ctx: (torch.empty(T, top, dtype=torch.int32, device="meta"), torch.empty(T, top, device="meta"))
    part._grouped = SimpleNamespace(takes=lambda ctx: not ctx.decode and T * top >= 512, run=lambda *a: calls.append("sorted"))
    ctx = SimpleNamespace(n_tokens=T, ws=Workspace(torch.device("meta")), seq_of_token=None, decode=decode)
    part._routed(torch.empty(T, W, dtype=torch.bfloat16, device="meta"), torch.empty(T, W, device="meta"), ctx)
    if "sorted" in calls:
        return "sorted"
    return {"moe_grouped": "one launch", "moe_expert_mma": "mma", "moe_gate_up": "cores"}[next(c for c in calls if c != "moe_place_gather" and c != "moe_gather")]


@pytest.mark.parametrize("E,W,F,top,T,sorted_us,one_launch_us", [
    # measured, us a layer
    (16, 4096, 2048, 2, 2048, 712, 300), (8, 4096, 8192, 2, 256, 462, 298), (2, 2048, 8192, 2, 2048, 583, 342), (4, 4096, 14336, 2, 4096, 2946, 2309),
    (64, 2048, 768, 2, 8192, 1907, 392), (8, 1024, 512, 2, 8192, 300, 235), (128, 2048, 768, 8, 2048, 3338, 438),
    (8, 1024, 512, 2, 16384, 441, 675)])
def test_the_sorted_form_only_where_it_is_quicker(monkeypatch, E, W, F, top, T, sorted_us, one_launch_us):
    assert route(monkeypatch, E, W, F, top, T) == ("sorted" if sorted_us < one_launch_us else "one launch")


def test_forms_at_the_limits(monkeypatch):
    assert route(monkeypatch, 1025, 512, 512, 2, 64) == "mma"                     # more experts than the one launch keeps ranges for
    assert route(monkeypatch, 1025, 512, 512, 2, 8192) == "sorted"                # more pairs than the mma.sync kernel takes
    assert route(monkeypatch, 16, 2048, 1024, 2, 250, decode=True) == "one launch"
    assert route(monkeypatch, 16, 2048, 1024, 2, 10000) == "sorted"
    assert route(monkeypatch, 16, 2048, 1024, 2, 10000, decode=True) == "cores"   # (a step that may not read back)


@pytest.mark.parametrize("E,W,F,top,T,mma_us,one_launch_us", [
    # measured, us a layer
    (4, 64, 64, 1, 16, 8.8, 14.7), (4, 64, 64, 1, 128, 11.4, 15.0), (8, 128, 128, 2, 16, 10.8, 16.1), (32, 256, 256, 2, 4, 14.6, 17.9),
    (128, 256, 128, 1, 61, 14.3, 19.3), (1000, 256, 128, 1, 8, 19.2, 22.2), (8, 512, 256, 2, 4, 20.2, 18.4), (128, 1024, 512, 1, 16, 39.9, 24.6), (4, 64, 64, 1, 256, 17.5, 15.7)])
def test_small_experts(monkeypatch, E, W, F, top, T, mma_us, one_launch_us):
    assert route(monkeypatch, E, W, F, top, T) == ("mma" if mma_us < one_launch_us else "one launch")
