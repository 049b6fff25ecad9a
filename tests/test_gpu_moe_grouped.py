"""The routed experts in one tcgen05 launch (csrc/moe_grouped.cu): row counts around the tiles' edges, experts without rows,
choices without an expert, widths that no tile divides, against float64."""
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,top,W,F", [(1, 4, 1, 64, 64), (8, 16, 2, 256, 128), (5, 3, 3, 72, 40), (33, 7, 2, 136, 72),
                                         (129, 2, 1, 64, 200), (300, 5, 2, 128, 328), (700, 4, 2, 512, 256)])
@pytest.mark.parametrize("on_input", [False, True])
def test_grouped_products(T, E, top, W, F, on_input):
    from gogguf_b200.csrc import kernels as K
    from gogguf_b200.csrc.tcgen05_gemm import check_status
    g = torch.Generator().manual_seed(T + E)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)          # noqa: E731
    h, w_gu, w_d = bf(T, W), bf(E, 2, F, W) * 0.2, bf(E, W, F) * 0.2
    idx = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32)
    idx[idx == E - 2] = -1 if T % 2 else 0                       # an expert without rows; choices without an expert
    wts = torch.rand(T, top, generator=g) + 0.2
    P, limit, slope, scale = T * top, 3.0, 1.702, 0.7
    d = lambda t: t.cuda()                                                      # noqa: E731
    offsets, place = torch.full((E + 1,), -7, dtype=torch.int32).cuda(), torch.full((P,), -7, dtype=torch.int32).cuda()
    row_wts, xs = torch.zeros(P).cuda(), torch.zeros(P, W, dtype=torch.bfloat16).cuda()
    K.moe_place_gather(d(h), d(wts), d(idx), P, E, top, on_input, offsets, place, row_wts, xs)
    flat = idx.view(-1).long()
    order = torch.argsort(torch.where(flat < 0, torch.full_like(flat, E), flat), stable=True)
    want_place = torch.empty(P, dtype=torch.int32)
    want_place[order] = torch.arange(P, dtype=torch.int32)
    assert torch.equal(place.cpu(), want_place)
    assert torch.equal(offsets.cpu().long(), torch.tensor([int(((flat >= 0) & (flat < e)).sum()) for e in range(E + 1)]))
    assert torch.equal(row_wts.cpu(), wts.view(-1)[order])
    y = torch.full((P, F), float("nan"), dtype=torch.bfloat16).cuda()
    K.moe_grouped(xs, d(w_gu), offsets, P, y, True, limit, slope, scale, None if on_input else row_wts)
    rows = torch.full((P, W), float("nan")).cuda()
    K.moe_grouped(y, d(w_d), offsets, P, rows, False)
    check_status(rows.device)
    res = torch.randn(T, W, generator=g)
    got = d(res)
    K.moe_combine(rows, place, got, T, top, None, idx=d(idx))
    want = res.double().clone()
    for p in range(P):
        e, t = int(flat[p]), p // top
        if e < 0:
            continue
        x = h[t].float() * wts.view(-1)[p] if on_input else h[t].float()
        x = x.to(torch.bfloat16).double()
        ge, u = (w_gu[e, 0].double() @ x).clamp(max=limit), (w_gu[e, 1].double() @ x).clamp(-limit, limit)
        a = ge * torch.sigmoid(slope * ge) * (u + 1.0) * scale * (1.0 if on_input else wts.view(-1)[p].double())
        ae = y[place[p].long()].cpu().double()
        assert (ae - a).abs().max() <= 2.0 ** -8 * a.abs().max() + 1e-5          # one rounding to bfloat16
        want[t] += w_d[e].double() @ ae
    assert rel_err(got.cpu(), want) < 1e-5                       # float32 sums of exact products


@pytest.mark.parametrize("T,W,E", [(1, 5, 3), (3, 72, 8), (600, 72, 9), (601, 300, 17), (80, 3100, 64)])
def test_router_logits_by_four_tokens(T, W, E):
    """A CTA of four tokens gives the bits of a CTA of one, against float64."""
    from gogguf_b200.csrc import kernels as K
    g = torch.Generator(device="cuda").manual_seed(W)
    for ht, wt in ((torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32), (torch.bfloat16, torch.float32)):
        h, wr = torch.randn(T, W, device="cuda", generator=g).to(ht), torch.randn(E, W, device="cuda", generator=g).to(wt)
        z, one = torch.empty(T, E, device="cuda"), torch.empty(1, E, device="cuda")
        K.moe_router_logits(h, wr, z, T)
        assert rel_err(z.cpu(), (h.double() @ wr.double().T).cpu()) < 1e-6
        K.moe_router_logits(h[T - 1:].contiguous(), wr, one, 1)
        assert torch.equal(one[0], z[T - 1])


# 17, 63 and 64 pairs (the ring with 64 rows of x); many experts, most of them empty; and so many tiles that every CTA of the
# persistent grid walks over three and more, over several experts, in the narrow form (more than 3 x 296) and in the wide one (3 x 148)
@pytest.mark.parametrize("T,E,top,W,F,limit", [(17, 5, 1, 64, 136, 7.0), (21, 6, 3, 128, 64, float("inf")), (64, 3, 1, 72, 200, float("inf")),
                                               (40, 300, 2, 64, 64, 7.0), (9, 1000, 8, 64, 72, float("inf")), (600, 1024, 2, 64, 64, 7.0),
                                               (40, 9, 1, 64, 12808, float("inf")), (300, 6, 2, 136, 6400, 7.0),
                                               (600, 4, 1, 64, 14000, float("inf")), (700, 5, 2, 200, 6464, 3.0)])
def test_many_tiles_and_experts(T, E, top, W, F, limit):
    from gogguf_b200.csrc import kernels as K
    from gogguf_b200.csrc.tcgen05_gemm import check_status
    g = torch.Generator(device="cuda").manual_seed(T + E)
    bf = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)          # noqa: E731
    h, w_gu, w_d = bf(T, W), bf(E, 2, F, W) * 0.2, bf(E, W, F) * 0.05
    idx = torch.rand(T, E, device="cuda", generator=g).topk(top, dim=-1).indices.to(torch.int32)
    idx[idx % 4 == 1] = 0 if top == 1 else -1                     # a quarter of the experts without rows
    flat, wts, P = idx.view(-1), torch.rand(T, top, device="cuda", generator=g) + 0.2, T * top
    i32 = lambda n: torch.empty(n, dtype=torch.int32, device="cuda")                        # noqa: E731
    offsets, place, row_wts, xs = i32(E + 1), i32(P), torch.empty(P, device="cuda"), torch.empty(P, W, device="cuda", dtype=torch.bfloat16)
    K.moe_place_gather(h, wts.view(-1), flat, P, E, top, False, offsets, place, row_wts, xs)
    y = torch.full((P, F), float("nan"), device="cuda", dtype=torch.bfloat16)
    K.moe_grouped(xs, w_gu, offsets, P, y, True, limit, 1.0, 0.7, row_wts, up_offset=0.0)
    rows = torch.full((P, W), float("nan"), device="cuda")
    K.moe_grouped(y, w_d, offsets, P, rows, False)
    check_status(rows.device)
    off = offsets.tolist()
    assert off[0] == 0 and off[E] == int((flat >= 0).sum())
    for e in torch.unique(flat[flat >= 0]).tolist():
        at = place[flat == e].long()
        assert sorted(at.tolist()) == list(range(off[e], off[e + 1]))
        x = h[torch.nonzero(flat == e)[:, 0] // top].double()
        ga, up = x @ w_gu[e, 0].double().T, x @ w_gu[e, 1].double().T
        a = ga.clamp(max=limit) * torch.sigmoid(ga.clamp(max=limit)) * up.clamp(-limit, limit) * 0.7 * wts.view(-1)[flat == e].double()[:, None]
        got = y[at].double()
        # (one rounding to bfloat16, and float32 sums behind an exponential)
        assert ((got - a).abs() <= 2.0 ** -8 * a.abs() + 1e-5 * a.abs().max()).all()
        want = got @ w_d[e].double().T
        # (the accumulator loses up to 2^-23 of itself with each of the F / 16 additions, half that on average, and always towards zero)
        assert rel_err(rows[at].double(), want) < 2e-6 + F / 16 * 2.0 ** -24
