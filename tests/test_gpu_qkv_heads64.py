"""The q/k/v product with heads of 64 in its epilogue (csrc/gemm_tcgen05.cu): norm, rotation and cache write of two heads per weight tile,
odd numbers of heads, tiles with heads of two kinds, against float64 and against the product and the kernel it stands for."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 8, 16, 17, 40, 64, 100, 128])
@pytest.mark.parametrize("nq,nkv,K_", [(16, 8, 1024), (3, 1, 136), (5, 3, 264), (2, 2, 2048), (1, 1, 72)])
@pytest.mark.parametrize("norm,fold", [(True, True), (False, False)])
def test_heads_of_64(M, nq, nkv, K_, norm, fold):
    from gogguf_b200.csrc import kernels as K, tcgen05_gemm as tc
    d, ps, dev = 64, 64, "cuda"
    g = torch.Generator(device=dev).manual_seed(M + nq)
    x = (torch.randn(M, K_, device=dev, generator=g) * 2).bfloat16()
    w = (torch.randn((nq + 2 * nkv) * d, K_, device=dev, generator=g) / math.sqrt(K_)).bfloat16()
    ssq = torch.rand(M, (K_ + 127) // 128, device=dev, generator=g) * 100 + 60 if fold else None
    qw, kw = ((1 + 0.2 * torch.randn(d, device=dev, generator=g)) if norm else None for _ in range(2))
    nseq = max(1, M // 5)
    seq = torch.tensor([t % nseq for t in range(M)], dtype=torch.int32, device=dev)
    pos = torch.tensor([60 + t // nseq for t in range(M)], dtype=torch.int32, device=dev)
    if M > 1:
        seq[-1] = -1
    table = torch.randperm(nseq * 3, generator=torch.Generator().manual_seed(1)).int().view(nseq, 3).to(dev)
    inv = torch.pow(torch.tensor(1e4, dtype=torch.float64), -2.0 * torch.arange(32, dtype=torch.float64) / d).to(dev)
    cos, sin = torch.empty(M, 32, device=dev), torch.empty(M, 32, device=dev)
    K.rope_tables(pos, inv, cos, sin)
    empty = 2.0 ** 100                                     # a value no product reaches marks what nobody wrote
    pools = [torch.full((nseq * 3, nkv, ps, d), empty, device=dev, dtype=torch.bfloat16) for _ in range(4)]
    qkv = torch.empty(M, (nq + 2 * nkv) * d, device=dev, dtype=torch.bfloat16)
    tc.gemm_tc_norm(x, w, qkv, in_ssq=ssq, eps=2e-6)
    q1 = torch.empty(M, nq * d, device=dev, dtype=torch.bfloat16)
    K.qk_norm_rope_cache(qkv, q1, qw, kw, 1e-5, cos, sin, pos, seq, table, ps, pools[0], pools[1], M, nq, nkv, d, d)
    q2 = torch.full((M + 1, nq * d), empty, device=dev, dtype=torch.bfloat16)
    tc.gemm_tc_qkv_rope(x, w, M, q2[:M], qw, kw, 1e-5, cos, sin, pos, seq, table, ps, pools[2], pools[3], nq, nkv, in_ssq=ssq, in_eps=2e-6, head_dim=64)
    tc.check_status(torch.device("cuda", 0))
    assert (q2[M] == empty).all() and all(torch.equal(a == empty, b == empty) for a, b in zip(pools[:2], pools[2:]))
    full = x.double() @ w.double().T
    if fold:
        full = full / torch.sqrt(ssq.double().sum(1, keepdim=True) / K_ + 2e-6)
    heads = full.view(M, nq + 2 * nkv, d)

    def turned(h, weight):
        if weight is not None:
            h = h / torch.sqrt((h ** 2).mean(-1, keepdim=True) + 1e-5) * weight.double()
        c, s = cos.double()[:, None], sin.double()[:, None]
        return torch.cat([h[..., :32] * c - h[..., 32:] * s, h[..., :32] * s + h[..., 32:] * c], -1)

    def close(got, want):                                  # (one rounding to bfloat16, and the sums' in 32 bits)
        return float((got.double() - want).norm() / want.norm()) < 2.0 ** -8

    assert close(q2[:M], turned(heads[:, :nq], qw).reshape(M, -1))
    live = [t for t in range(M) if int(seq[t]) >= 0]
    for pool, want in ((pools[2], turned(heads[:, nq:nq + nkv], kw)), (pools[3], heads[:, nq + nkv:])):
        if live:
            got = torch.stack([pool[table[seq[t], pos[t] // ps].long(), :, int(pos[t]) % ps] for t in live])
            assert close(got, want[live])
