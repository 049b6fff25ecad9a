"""Forms with 16-byte accesses against the element forms they take the place of: retention in chunks (csrc/retention.cu) against
the token-by-token scan, q/k preparation with a partial rotation (csrc/elementwise.cu) against float64."""
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("d,dv,rot", [(128, 128, 32), (64, 64, 64), (32, 40, 8), (96, 128, 0), (128, 72, 128), (64, 128, 20)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_retention_chunks(d, dv, rot, dt):
    from gogguf_b200.csrc import kernels as K
    g = torch.Generator(device=DEV).manual_seed(d + dv)
    lens, H = [1, 64, 65, 130, 63], 3
    T, n = sum(lens), len(lens)
    x = torch.randn(T, 2 * H * (d + dv), device=DEV, generator=g).to(dt)
    ang = torch.rand(T, max(rot // 2, 1), device=DEV, generator=g) * 6
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    cu = i32([sum(lens[:i]) for i in range(n + 1)])
    sot, slots = i32([i for i, m in enumerate(lens) for _ in range(m)]), i32([3, 0, 5, 1, 2])
    decay = torch.tensor([0.9, 0.99, 1.0], device=DEV)
    start = torch.randn(6, H, d, dv, device=DEV, generator=g) * 0.1
    both = []
    for chunks in (False, True):
        state, out = start.clone(), torch.full((T, H * dv), float("nan"), device=DEV, dtype=dt)
        if chunks:
            scratch = torch.empty(K.retention_chunks_scratch(T, n, H, d, dv), device=DEV)
            K.retention_chunks(x, out, scratch, state, cos, sin, cu, slots, sot, decay, T, n, H, d, dv, rot, d ** -0.5, 1e-5, 1.3)
        else:
            raw = torch.empty(T, H * dv, device=DEV)
            K.retention(x, out, raw, state, cos, sin, cu, slots, sot, decay, T, n, H, d, dv, rot, d ** -0.5, 1e-5, 1.3, 0)
        both.append((out.float(), state))
    (a, sa), (b, sb) = both
    # (float32 sums in another order; an output in bfloat16 may round to its other neighbour)
    assert rel_err(b, a) < (3e-5 if dt == torch.float32 else 2.0 ** -7) and rel_err(sb, sa) < 3e-5
    assert torch.equal(sb[4], start[4])


@pytest.mark.parametrize("d,rot", [(128, 64), (128, 16), (64, 32), (64, 0), (256, 96), (128, 112), (128, 128)])
@pytest.mark.parametrize("normed", [True, False])
def test_partial_rotation(d, rot, normed):
    from gogguf_b200.csrc import kernels as K
    g = torch.Generator(device=DEV).manual_seed(d + rot)
    T, nq, nkv, ps = 37, 5, 2, 16
    x = torch.randn(T, (nq + 2 * nkv) * d, device=DEV, generator=g).to(torch.bfloat16)
    x[3, rot + 1 if rot < d else 0] = float("inf") if rot < d - 2 and not normed else 1.0     # stays where it is
    qw, kw = ((1 + 0.1 * torch.randn(d, device=DEV, generator=g)) for _ in range(2)) if normed else (None, None)
    ang = torch.rand(T, max(rot // 2, 1), device=DEV, generator=g) * 6
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    kp, vp = (torch.full((4, nkv, ps, d), -7.0, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    pos, sot = i32(list(range(T))), i32([0] * (T - 1) + [-1])
    table = i32([[2, 0, 3]])
    q = torch.full((T, nq * d), float("nan"), device=DEV, dtype=torch.bfloat16)
    K.qk_norm_rope_cache(x, q, qw, kw, 1e-5, cos, sin, pos, sot, table, ps, kp, vp, T, nq, nkv, d, rot)
    h = x.double().view(T, nq + 2 * nkv, d)

    def prepared(v, w):
        v = v / (v.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() if w is not None else v.clone()
        a, b, r = v[..., :rot // 2].clone(), v[..., rot // 2:rot].clone(), rot // 2
        c, s = (t.double()[:, None, :r] for t in (cos, sin))
        v[..., :r], v[..., r:rot] = a * c - b * s, a * s + b * c
        return v

    def close(got, want):
        got, fin = got.double(), torch.isfinite(want)
        assert torch.equal(got[~fin], want[~fin])
        assert ((got - want)[fin].abs() <= 2.0 ** -8 * want[fin].abs() + 1e-5 * want[fin].abs().max()).all()

    close(q.view(T, nq, d), prepared(h[:, :nq], qw))
    k, v = prepared(h[:, nq:nq + nkv], kw), h[:, nq + nkv:]
    for t in range(T - 1):
        page = int(table[0, t // ps])
        close(kp[page, :, t % ps], k[t])
        close(vp[page, :, t % ps], v[t])
    assert float(kp[1].float().max()) == -7.0 and float(kp[3, :, (T - 1) % ps].float().max()) == -7.0      # padding wrote nothing
