"""The plain matrix product's tile sizes (csrc/gemm_plain.cu): every number of rows at which another tile is taken, ragged
sizes, strides and alignments, against float64; and the promise that a row's bits do not depend on the rows beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def K():
    from gogguf_b200.csrc import kernels
    return kernels


# (a float32 sum of K products in four slices: rounding grows like sqrt(K / 4) 2^-24, three times that as the bound)
def bound(k):
    return 3.0 * (k ** 0.5 / 2 + 4) * 2.0 ** -24


@pytest.mark.parametrize("N,K_", [(16, 4), (130, 36), (49, 129), (2048, 260), (700, 1800), (2500, 96), (5000, 200)])
@pytest.mark.parametrize("dtypes", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32)])
def test_rows_of_every_tile(N, K_, dtypes):
    g = torch.Generator(device="cuda").manual_seed(3)
    wide = torch.randn(700, K_ + 8, device="cuda", generator=g).to(dtypes[0])
    w = torch.randn(N, K_, device="cuda", generator=g).to(dtypes[1])
    bias = torch.randn(N, device="cuda", generator=g)
    first = None
    for off in (0, 1):                          # (rows that start off a 16-byte boundary take element loads)
        x = wide[:, off:off + K_]
        for M in (1, 2, 3, 4, 5, 8, 9, 12, 16, 17, 32, 33, 65, 129, 300, 700):
            out = torch.full((M, N), float("nan"), device="cuda")
            K().gemm_plain(x[:M], w, out)
            want = x[:M].double() @ w.double().T
            assert (out.double() - want).norm() <= bound(K_) * (x[:M].double().abs() @ w.double().abs().T).norm()
            if M == 1:
                first = out[0].clone()
            assert torch.equal(out[0], first)
            res = torch.randn(M, N, device="cuda", generator=g)
            acc = res.clone()
            K().gemm_plain(x[:M], w, acc, accumulate=True, bias=bias)
            assert torch.equal(acc, res + (out + bias))


@pytest.mark.parametrize("pos", [0, 7, 8, 63, 64, 65, 517])
def test_attention_keys_in_groups(pos):
    """Contexts around the groups of eight keys and the eight warps that share them, against float64."""
    g = torch.Generator(device="cuda").manual_seed(9)
    nq, nkv, d, ps = 4, 2, 40, 16
    pages = pos // ps + 1
    q = torch.randn(1, nq, d, device="cuda", generator=g)
    kp, vp = (torch.randn(pages, nkv, ps, d, device="cuda", generator=g) for _ in range(2))
    table = torch.arange(pages - 1, -1, -1, device="cuda", dtype=torch.int32).view(1, pages)
    out = torch.empty(1, nq, d, device="cuda")
    for window in (0, 5):
        K().attention_plain(q, kp, vp, out, torch.tensor([pos], device="cuda", dtype=torch.int32),
                            torch.zeros(1, device="cuda", dtype=torch.int32), table, ps, 1, nq, nkv, d, d ** -0.5, window)
        lo = max(0, pos - window + 1) if window else 0
        order = table[0].long()
        keys, vals = (t[order].transpose(0, 1).reshape(nkv, -1, d)[:, lo:pos + 1].double().repeat_interleave(2, 0) for t in (kp, vp))
        p = torch.softmax(torch.einsum("hd,hkd->hk", q[0].double(), keys) * d ** -0.5, -1)
        want = torch.einsum("hk,hkd->hd", p, vals)
        # (a weight's relative error is the score's absolute one: d terms of size about 1, three times their rounding)
        assert (out[0].double() - want).abs().max() <= 3 * (d + 8) * 2.0 ** -24 * vals.abs().max()


@pytest.mark.parametrize("d,dv", [(128, 128), (120, 64), (36, 132), (256, 256), (30, 30)])
def test_attention_head_sizes(d, dv):
    """Lanes with four columns and one or two groups of them, sizes that leave lanes without columns, element loads."""
    g = torch.Generator(device="cuda").manual_seed(d)
    nq, nkv, ps, pos = 2, 1, 64, 150
    for dt, tol in ((torch.float32, 3 * (d + 8) * 2.0 ** -24), (torch.bfloat16, 2.0 ** -8)):
        q = torch.randn(1, nq, d, device="cuda", generator=g).to(dt)
        kp, vp = (torch.randn(3, nkv, ps, n, device="cuda", generator=g).to(dt) for n in (d, dv))
        table = torch.tensor([[2, 0, 1]], device="cuda", dtype=torch.int32)
        out = torch.empty(1, nq, dv, device="cuda", dtype=dt)
        K().attention_plain(q, kp, vp, out, torch.tensor([pos], device="cuda", dtype=torch.int32),
                            torch.zeros(1, device="cuda", dtype=torch.int32), table, ps, 1, nq, nkv, d, d ** -0.5, 0, dv=dv)
        keys, vals = (t[[2, 0, 1], 0].reshape(-1, t.shape[-1])[:pos + 1].double() for t in (kp, vp))
        want = torch.softmax(q[0].double() @ keys.T * d ** -0.5, -1) @ vals
        assert (out[0].double() - want).abs().max() <= tol * vals.abs().max()


@pytest.mark.parametrize("dtypes", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("N,K_,off", [(70, 33, 0), (1000, 129, 0), (333, 260, 1), (5000, 67, 0), (2100, 64, 0)])
def test_rows_by_elements(N, K_, off, dtypes):
    """Rows off their boundaries and bfloat16 matrices in the tiles of more than 16 rows: element copies, values kept as they lie in
    memory; outputs in bfloat16 and behind a stride."""
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(1300, K_ + 7, device="cuda", generator=g).to(dtypes[0])[:, off:off + K_]
    w = torch.randn(N, K_, device="cuda", generator=g).to(dtypes[1])
    first = None
    for M in (1, 31, 63, 64, 65, 128, 300, 610, 1300):
        wide = torch.full((M, N + 3), -7.0, device="cuda")
        K().gemm_plain(x[:M], w, wide[:, :N])
        out = wide[:, :N]
        want = x[:M].double() @ w.double().T
        assert (out.double() - want).norm() <= bound(K_) * (x[:M].double().abs() @ w.double().abs().T).norm()
        first = out[0].clone() if first is None else first
        assert torch.equal(out[0], first) and (wide[:, N:] == -7.0).all()
        half = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        K().gemm_plain(x[:M], w, half)
        assert torch.equal(half, out.to(torch.bfloat16))
