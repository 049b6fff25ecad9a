"""What the CTA-pair product stores (csrc/gemm_tcgen05.cu): the partial tiles of a split, which leave by whole lines, and, thread by row,
bfloat16 and float32 rows, sums into the residual and gated units; rows that end inside a warp's 32, columns inside a
chunk, rows off a 16-byte boundary, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split,M,N,K", [
    (False, 129, 264, 64), (False, 157, 331, 2048), (False, 300, 1000, 2048), (False, 333, 2056, 1024), (False, 566, 4096, 512), (False, 600, 300, 1600),
    (True, 157, 331, 2048), (True, 300, 1000, 2048), (True, 333, 2056, 1024), (True, 600, 300, 1600)])
def test_rows_by_lines(M, N, K, split):
    from gogguf_b200.csrc import tcgen05_gemm as tc
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = (torch.randn(n, K, device="cuda", generator=g).to(torch.bfloat16) for n in (M, N))
    want = x.double() @ w.double().T
    room = tc.pair_scratch_elems(M, N, K)
    assert room > 0 or not split                         # (a plan that no longer splits would leave this case without its subject)
    scratch = torch.empty(room, device="cuda") if split else None
    size = want.norm()
    for pad in (0, 3):                                   # rows whose start is on no 16-byte boundary
        bf = torch.full((M, N + pad), -7.0, device="cuda", dtype=torch.bfloat16)
        tc.gemm_tc(x, w, bf[:, :N], scratch=scratch, cluster=True)
        f32 = torch.full((M, N + pad), -7.0, device="cuda")
        tc.gemm_tc(x, w, f32[:, :N], scratch=scratch, cluster=True)
        res = torch.randn(M, N + pad, device="cuda", generator=g)
        acc = res.clone()
        tc.gemm_tc(x, w, acc[:, :N], accumulate=True, scratch=scratch, cluster=True)
        tc.check_status(x.device)
        # (float32 sums of K products, K / 16 truncations of the accumulator; then one rounding to bfloat16)
        bound = 2e-6 + 2e-7 * K ** 0.5
        assert (f32[:, :N].double() - want).norm() <= bound * size
        assert (acc[:, :N].double() - res[:, :N].double() - want).norm() <= 2 * bound * size
        assert (bf[:, :N].double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()
        for t, before in ((bf, torch.full_like(bf, -7.0)), (f32, torch.full_like(f32, -7.0)), (acc, res)):
            assert torch.equal(t[:, N:], before[:, N:])  # nothing beyond a row's end


@pytest.mark.parametrize("M,I,K", [(130, 128, 128), (333, 576, 512), (290, 192, 2048)])
def test_gated_rows(M, I, K):
    from gogguf_b200.csrc import tcgen05_gemm as tc
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    gate, up = (torch.randn(I, K, device="cuda", generator=g).to(torch.bfloat16) * K ** -0.5 for _ in range(2))
    out = torch.full((M, I), float("nan"), device="cuda", dtype=torch.bfloat16)
    tc.gemm_tc(x, tc.interleave_gate_up(gate, up), out, cluster=True, swiglu=True)
    tc.check_status(x.device)
    a, b = x.double() @ gate.double().T, x.double() @ up.double().T
    want = a * torch.sigmoid(a) * b
    assert (out.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()
