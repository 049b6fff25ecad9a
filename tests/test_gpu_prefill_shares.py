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
