"""Prefill attention whose pages are shared by the CTAs of a cluster (csrc/attention_fast.cu): shares without pages, rows that
see none of a share, windows, head sizes between the templates', sinks and gates, against the unshared form and float64."""
import math

import pytest
import torch

from test_gpu_kernels import attention_reference, make_paged, rel, step_meta




@pytest.mark.gpu
@pytest.mark.parametrize("nq,nkv,d,window,seqs", [(4, 1, 128, 0, [(700, 330)]), (8, 2, 64, 0, [(64, 3), (900, 1), (130, 130)]),
                                                  (4, 2, 128, 100, [(1000, 200), (20, 20)]), (2, 1, 40, 0, [(333, 129)])])
@pytest.mark.parametrize("splits", [2, 3, 8])
def test_shared_pages(nq, nkv, d, window, seqs, splits):
    from gogguf_b200.csrc import fast_attention as fa
    from gogguf_b200.csrc import tcgen05_gemm as tc
    dev = torch.device("cuda")
    kp, vp, table, ks, vs = make_paged(seqs, nkv, d, torch.bfloat16, seed=9)
    pos, sot, cu, cl = step_meta(seqs)
    T = pos.numel()
    g = torch.Generator(device=dev).manual_seed(10)
    q = torch.randn(T, nq, d, device=dev, generator=g).to(torch.bfloat16)
    scale = 1.0 / math.sqrt(d)
    want = attention_reference(q, ks, vs, seqs, nq, nkv, scale, window)
    tiles = sum(-(-n // 128) for _, n in seqs)
    args = (q, kp, vp), (cu, cl, sot, table, 64, T, len(seqs), tiles, nq, nkv, d, scale, window)
    out = torch.full((T, nq, d), float("nan"), device=dev, dtype=torch.bfloat16)
    fa.attn_prefill_tc(*args[0], out, *args[1], splits=splits)
    tc.check_status(dev)
    assert rel(out, want) < 8e-3
    sink = torch.randn(nq, device=dev, generator=g)
    gate = torch.randn(T, nq * d, device=dev, generator=g).to(torch.bfloat16)
    for kw in (dict(sink=sink), dict(gate=gate, out_scale=0.7)):
        whole = torch.empty_like(out)
        fa.attn_prefill_tc(*args[0], whole, *args[1], **kw)
        out.fill_(float("nan"))
        fa.attn_prefill_tc(*args[0], out, *args[1], splits=splits, **kw)
        tc.check_status(dev)
        # (the two take their exponentials against other maxima: P rounds to bfloat16 elsewhere)
        assert rel(out, whole) < 8e-3


def test_how_many_shares():
    from gogguf_b200.csrc.fast_attention import prefill_splits
    assert prefill_splits(333, 1, 32, 6433) == 2 and prefill_splits(333, 1, 16, 6433) == 4 and prefill_splits(2048, 1, 32, 2048) == 1
    assert prefill_splits(10, 1, 32, 6000) == 8 and prefill_splits(10, 1, 32, 500) == 1 and prefill_splits(1, 1, 512, 8000) == 1


@pytest.mark.parametrize("tokens,seqs,nq,reach,max_new,wide,unshared,shared", [
    # measured: us unshared, us by the number of shares
    (333, 1, 16, 520, 333, 64, 10.35, {2: 14.83, 4: 13.35}), (128, 1, 16, 640, 128, 64, 10.79, {2: 15.62, 4: 12.74, 8: 12.04}),
    (128, 1, 8, 1300, 128, 64, 17.66, {2: 18.78, 4: 14.29, 8: 12.68}), (640, 1, 16, 1300, 640, 64, 17.92, {2: 19.83}),
    (1920, 3, 8, 1700, 640, 64, 21.93, {2: 24.78}), (333, 1, 32, 640, 333, 128, 12.38, {2: 14.89}), (128, 1, 64, 640, 128, 128, 12.84, {2: 13.87, 4: 14.18}),
    (333, 1, 24, 1700, 333, 128, 25.14, {2: 20.4, 4: 28.94}), (640, 1, 16, 704, 640, 128, 15.15, {2: 18.19}),
    (333, 1, 16, 6400, 333, 64, 66.91, {2: 43.52, 4: 31.12}), (3, 1, 32, 6400, 3, 128, 78.3, {2: 43.16, 4: 25.24, 8: 19.4})])
def test_shares_are_worth_their_sums(tokens, seqs, nq, reach, max_new, wide, unshared, shared):
    """The number of shares is never one that was measured slower than none (nor one that was not measured: more clusters than
    the device holds), and within a quarter of the quickest."""
    from gogguf_b200.csrc.fast_attention import prefill_splits
    took = {1: unshared, **shared}[prefill_splits(tokens, seqs, nq, reach, max_new, wide)]
    assert took <= unshared and took <= 1.25 * min(unshared, *shared.values())
