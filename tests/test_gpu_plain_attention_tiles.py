"""32-bit attention over tiles of rows and over shares of the keys (csrc/attention_plain.cu): sequences of unequal lengths behind histories,
windows, chunks, sinks, gates, head sizes and groups, against float64; what a token may not see is not read into its sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def run(new, ctx, nq, nkv, d, dv, ps, tiles, seed=3, **kw):
    from gogguf_b200.csrc import kernels as K
    g = torch.Generator(device="cuda").manual_seed(seed)
    R = lambda *s: torch.randn(*s, device="cuda", generator=g)                                       # noqa: E731
    T, B = sum(new), len(new)
    width = max((c + n + ps - 1) // ps for c, n in zip(ctx, new)) + 1
    order = torch.randperm(B * width, device="cuda", generator=g).to(torch.int32).view(B, width)
    kp, vp = R(B * width, nkv, ps, d), R(B * width, nkv, ps, dv)
    for b in range(B):                                   # nothing lies behind the sequences' ends
        flat = order[b].long()
        for pool in (kp, vp):
            t = pool[flat].transpose(1, 2).reshape(width * ps, nkv, -1)
            t[ctx[b] + new[b]:] = float("nan")
            pool[flat] = t.view(width, ps, nkv, -1).transpose(1, 2)
    q = R(T, nq, d)
    sink = R(nq) if kw.get("sink") else None
    gate = R(T, nq * dv) if kw.get("gate") else None
    pos = torch.cat([torch.arange(c, c + n) for c, n in zip(ctx, new)]).int().cuda()
    seq = torch.cat([torch.full((n,), b) for b, n in enumerate(new)]).int().cuda()
    cu = torch.tensor([0] + [sum(new[:i + 1]) for i in range(B)], dtype=torch.int32, device="cuda")
    out = torch.full((T, nq, dv), float("nan"), device="cuda")
    window, chunk = kw.get("window", 0), kw.get("chunk", 0)
    K.attention_plain(q, kp, vp, out, pos, seq, order, ps, T, nq, nkv, d, d ** -0.5, window, dv=dv, sink=sink, out_scale=0.7, chunk=chunk,
                      gate=gate, cu_seqlens=cu if tiles else None, n_seqs=B if tiles else 0)
    for b in range(B):
        keys, vals = (pool[order[b].long()].transpose(1, 2).reshape(width * ps, nkv, -1).double().repeat_interleave(nq // nkv, 1) for pool in (kp, vp))
        rows = slice(int(cu[b]), int(cu[b + 1]))
        n = ctx[b] + new[b]
        s = torch.einsum("thd,khd->htk", q[rows].double(), keys[:n]) * d ** -0.5
        i, j = pos[rows].long()[:, None], torch.arange(n, device="cuda")[None]
        hide = j > i
        if window:
            hide = hide | (i - j >= window)
        if chunk:
            hide = hide | (j < i // chunk * chunk)
        s = s.masked_fill(hide, -float("inf"))
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None, None].expand(nq, s.shape[1], 1)], -1)
        p = torch.softmax(s, -1)[..., :n]
        want = torch.einsum("htk,khd->thd", p, vals[:n]) * 0.7
        if gate is not None:
            want = want * torch.sigmoid(gate[rows].double()).view(-1, nq, dv)
        # (a weight's relative error is the score's absolute one: d terms of size about 1, three times their rounding)
        assert (out[rows].double() - want).abs().max() <= 3 * (d + 8) * 2.0 ** -24 * vals[:n].abs().max(), (b, kw)


@pytest.mark.parametrize("tiles", [True, False])
@pytest.mark.parametrize("opts", [{}, dict(window=7), dict(window=33, sink=True), dict(chunk=40, gate=True), dict(sink=True, gate=True)])
@pytest.mark.parametrize("nq,nkv,d,dv,ps", [(4, 2, 128, 128, 64), (3, 3, 36, 64, 16), (6, 2, 120, 120, 64), (2, 1, 4, 4, 64), (8, 1, 64, 100, 64)])
def test_prompts_and_turns(nq, nkv, d, dv, ps, opts, tiles):
    run([33, 1, 70, 16, 5], [0, 30, 61, 0, 100], nq, nkv, d, dv, ps, tiles, **opts)


@pytest.mark.parametrize("new,ctx", [([31], [0]), ([32], [1]), ([16, 16], [0, 700]), ([150], [33])])
def test_edges_of_tiles(new, ctx):
    run(new, ctx, 2, 1, 32, 32, 64, True)


@pytest.mark.parametrize("B,nq,ctx", [(1, 2, 1000), (3, 4, 555), (4, 16, 700), (1, 1, 63), (7, 8, 64), (2, 4, 5)])
@pytest.mark.parametrize("d,dv", [(128, 128), (256, 36), (30, 30)])
def test_shares_of_the_keys(B, nq, ctx, d, dv):
    run([1] * B, [max(0, ctx - 37 * i) for i in range(B)], nq, 1, d, dv, 64, False, sink=True, gate=True)
    run([1] * B, [max(0, ctx - 37 * i) for i in range(B)], nq, 1, d, dv, 64, False, window=130)


def test_an_infinity_behind_a_token_stays_there():
    from gogguf_b200.csrc import kernels as K
    g = torch.Generator(device="cuda").manual_seed(1)
    q, kp, vp = torch.randn(40, 2, 32, device="cuda", generator=g), torch.randn(1, 1, 64, 32, device="cuda", generator=g), torch.randn(1, 1, 64, 32, device="cuda", generator=g)
    vp[0, 0, 20] = float("inf")
    out = torch.empty(40, 2, 32, device="cuda")
    K.attention_plain(q, kp, vp, out, torch.arange(40, device="cuda", dtype=torch.int32), torch.zeros(40, device="cuda", dtype=torch.int32),
                      torch.zeros(1, 1, device="cuda", dtype=torch.int32), 64, 40, 2, 1, 32, 1.0, 0,
                      cu_seqlens=torch.tensor([0, 40], device="cuda", dtype=torch.int32), n_seqs=1)
    assert out[:20].isfinite().all() and not out[20:].isfinite().any()


def test_an_infinity_with_a_weight_of_zero():
    """A value that a row sees counts also where its weight is too small for a float32, in tiles on an edge and inside, as a row at a time."""
    from gogguf_b200.csrc import kernels as K
    g = torch.Generator(device="cuda").manual_seed(4)
    T, ints = 100, dict(device="cuda", dtype=torch.int32)
    q, kp, vp = torch.ones(T, 2, 32, device="cuda"), torch.zeros(2, 1, 64, 32, device="cuda"), torch.randn(2, 1, 64, 32, device="cuda", generator=g)
    for at in (5, 90):                                     # scores 200 below the others
        kp[at // 64, 0, at % 64] = -200.0 / 32
        vp[at // 64, 0, at % 64] = float("inf")
    outs = []
    for cu in (None, torch.tensor([0, T], **ints)):
        outs.append(torch.empty(T, 2, 32, device="cuda"))
        K.attention_plain(q, kp, vp, outs[-1], torch.arange(T, **ints), torch.zeros(T, **ints), torch.tensor([[0, 1]], **ints), 64, T, 2, 1, 32,
                          1.0, 0, cu_seqlens=cu, n_seqs=1)
    assert torch.equal(outs[0].isfinite(), outs[1].isfinite())
    assert outs[0][:5].isfinite().all() and not outs[0][5:].isfinite().any()
