"""The 32-bit product on the tensor cores (csrc/gemm_f32_parts.cu): every tile and edge of it, shares of K, rows off 16-byte
boundaries, infinities and NaN, and an error against 64 bits no larger than that of the multiply-adds of the plain product."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TILES = (32, 64, 96, 128, 160, 192)


def K():
    from gogguf_b200.csrc import kernels
    return kernels


def parts(x, w, out, tile=-1, shares=0, **kw):
    M = kw.get("m") or x.shape[0]
    scratch = torch.full((K().f32_parts_scratch(M, w.shape[0], w.shape[1], tile, shares),), 255, dtype=torch.uint8, device="cuda")
    K().gemm_f32_parts(x, w, out, scratch, tile=tile, shares=shares, **kw)
    return out


def off(out, want):
    return float((out.double() - want).norm() / want.norm())


@pytest.mark.parametrize("tile", range(6))
@pytest.mark.parametrize("N,K_,shares", [(1, 4, 1), (127, 60, 1), (128, 64, 1), (130, 196, 2), (300, 1800, 3), (2048, 520, 1)])
def test_tiles_and_shares(tile, N, K_, shares):
    g = torch.Generator(device="cuda").manual_seed(N + K_)
    wide = torch.randn(400, K_ + 8, device="cuda", generator=g)
    w = torch.randn(N, K_, device="cuda", generator=g)
    bias = torch.randn(N, device="cuda", generator=g)
    for o, M in ((0, 1), (1, TILES[tile] - 1), (0, TILES[tile]), (1, TILES[tile] + 1), (0, 390)):
        x = wide[:, o:o + K_]
        room = torch.full((M + 1, N + 3), -7.0, device="cuda")
        parts(x, w, room[:M, :N], tile, shares, m=M)
        out = room[:M, :N]
        want = x[:M].double() @ w.double().T
        # (the parts left out are 2^-24 of a product, a sum of 32 columns is cut off twice at 2^-23, the sums of those are rounded)
        bound = (3 + (K_ / 32) ** 0.5 / 2) * 2.0 ** -23
        assert (out.double() - want).norm() <= bound * (x[:M].double().abs() @ w.double().abs().T).norm()
        assert (room[:, N:] == -7.0).all() and (room[M:] == -7.0).all()
        again = parts(x, w, torch.empty(M, N, device="cuda"), tile, shares, m=M)
        assert torch.equal(again, out)
        res = torch.randn(M, N, device="cuda", generator=g)
        acc = parts(x, w, res.clone(), tile, shares, m=M, accumulate=True, bias=bias)
        assert torch.equal(acc, res + (out + bias))


@pytest.mark.parametrize("M,N,K_", [(17, 2048, 2048), (64, 4096, 1024), (150, 1800, 1800), (450, 2048, 5376), (600, 1024, 3072), (333, 700, 12288)])
def test_error_is_no_larger_than_the_multiply_adds(M, N, K_):
    g = torch.Generator(device="cuda").manual_seed(M)
    for spread in (0.0, 3.0):                      # rows and columns of like size, and over some powers of ten
        x = torch.randn(M, K_, device="cuda", generator=g) * torch.exp(spread * torch.randn(K_, device="cuda", generator=g))
        w = torch.randn(N, K_, device="cuda", generator=g) * 0.02
        want = x.double() @ w.double().T
        plain = torch.empty(M, N, device="cuda")
        K().gemm_plain(x, w, plain)
        assert off(parts(x, w, torch.empty(M, N, device="cuda")), want) <= off(plain, want)


def low_bits(g, *shape):
    """Numbers whose significands lie just below 1 + 2^-7, of either sign and over some powers of two: cut off to 8 bits they would leave
    2^-7 of themselves, and that 2^-8 of itself."""
    n = 1 + 2.0 ** -7 - 2.0 ** -23 * torch.randint(1, 64, shape, device="cuda", generator=g)
    return n * torch.exp2(torch.randint(-9, 9, shape, device="cuda", generator=g).float()) * (1 - 2 * torch.randint(0, 2, shape, device="cuda", generator=g))


@pytest.mark.parametrize("tile,shares", [(0, 1), (2, 3), (5, 1)])
@pytest.mark.parametrize("draw", ["low bits", "any"])
def test_a_term_alone_keeps_its_bits(draw, tile, shares):
    """A row of x with one number in it: the output is that number's product."""
    g = torch.Generator(device="cuda").manual_seed(5)
    M, N, K_ = 200, 260, 448
    some = (lambda *s: low_bits(g, *s)) if draw == "low bits" else (lambda *s: torch.randn(*s, device="cuda", generator=g))
    at = torch.randint(0, K_, (M, 1), device="cuda", generator=g)
    x, w = torch.zeros(M, K_, device="cuda").scatter_(1, at, some(M, 1)), some(N, K_)
    want = x.double() @ w.double().T
    out = parts(x, w, torch.empty(M, N, device="cuda"), tile, shares)
    # what is left out of a product is 2^-24 of it, the two sums with the large parts are cut off at 2^-23 of it at most, of which one adds
    # nothing; the sums before them are 2^-7 of it and are cut off ten times
    assert ((out.double() - want).abs() <= (1 + 2 + 10 * 2.0 ** -6) * 2.0 ** -24 * want.abs()).all()


@pytest.mark.parametrize("K_", [512, 2048])
def test_terms_of_one_sign(K_):
    """Equal terms, whose losses add up if they have a sign."""
    c = 1 + 2.0 ** -7 - 2.0 ** -23
    x, w = torch.full((96, K_), c, device="cuda"), torch.full((384, K_), c, device="cuda")
    want = x.double() @ w.double().T
    e = (parts(x, w, torch.empty(96, 384, device="cuda")).double() - want).abs() / want
    # 2^-24 left out, a sum of 32 columns cut off twice at 2^-23 of it, and the rounding of K / 32 partial sums, none above 2^-24 of the last
    assert float(e.max()) <= (1 + 4) * 2.0 ** -24 + K_ / 64 * 2.0 ** -24


@pytest.mark.parametrize("shares", [1, 3])
def test_infinities_and_nan(shares):
    g = torch.Generator(device="cuda").manual_seed(2)
    M, N, K_ = 70, 200, 260
    x, w = torch.randn(M, K_, device="cuda", generator=g), torch.randn(N, K_, device="cuda", generator=g)
    inf = float("inf")
    x[3, 5], x[4, 7], x[5, 0], x[6, :] = inf, -inf, float("nan"), 0.0
    x[7, 9] = torch.tensor(0x7f800001, dtype=torch.int32).view(torch.float32).item()       # a NaN whose upper half is an infinity
    x[8, 11], x[9, 12] = 3.4e38, 2e38
    w[10, 12], w[11, 5], w[12, 130], w[13, 5] = 3.0, 0.0, inf, inf
    out, plain = parts(x, w, torch.empty(M, N, device="cuda"), shares=shares), torch.empty(M, N, device="cuda")
    K().gemm_plain(x, w, plain)
    assert torch.equal(out.isnan(), plain.isnan()) and torch.equal(out.isinf(), plain.isinf())
    assert torch.equal(out[out.isinf()], plain[plain.isinf()])
    fin = plain.isfinite()
    assert torch.allclose(out[fin], plain[fin], rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("o", [0, 1])
@pytest.mark.parametrize("tile", range(6))
def test_rows_that_are_not_finite(tile, o):
    """Whole rows of them, and operands beyond the largest bfloat16 number whose products are finite; rows of x on and off 16-byte boundaries."""
    g = torch.Generator(device="cuda").manual_seed(tile)
    M, N, K_ = 230, 140, 260
    x, w = torch.randn(M, K_ + 4, device="cuda", generator=g)[:, o:o + K_], torch.randn(N, K_, device="cuda", generator=g) * 0.01
    x[:, 100] = 3.4e38                                                     # rounds to an infinity in 8 bits
    w[:, 100] = torch.randn(N, device="cuda", generator=g) * 1e-38
    x[5:90:3, 7], x[6:200:7, 9] = float("nan"), float("inf")
    x[64:72, 255:] = float("nan")                                          # (the last columns, and whole groups of rows)
    w[17, 9], w[18, 9], res = 0.0, -1.0, torch.randn(M, N, device="cuda", generator=g)
    bias = torch.randn(N, device="cuda", generator=g)
    out, plain = parts(x, w, res.clone(), tile, accumulate=True, bias=bias), res.clone()
    K().gemm_plain(x, w, plain, accumulate=True, bias=bias)
    assert torch.equal(out.isnan(), plain.isnan()) and torch.equal(out.isinf(), plain.isinf())
    assert torch.equal(out[out.isinf()], plain[plain.isinf()])
    fin = plain.isfinite()
    want = (x.double() @ w.double().T + bias + res)[fin]
    mag = (x.double().abs() @ w.double().abs().T + bias.abs() + res.abs())[fin]
    assert fin.any() and ((out[fin].double() - want).abs() <= (K_ + 2) * 2.0 ** -24 * mag).all()     # (a chain of K multiply-adds)


def test_refusals():
    x, w, out = torch.zeros(4, 8, device="cuda"), torch.zeros(16, 8, device="cuda"), torch.zeros(4, 16, device="cuda")
    from gogguf_b200.csrc.build import KernelError
    s = torch.empty(1 << 16, dtype=torch.uint8, device="cuda")
    for args in ((x[:, :6], torch.zeros(16, 6, device="cuda"), out, s), (x, w, out, s[:64]), (x.bfloat16(), w, out, s), (x, w, out[:3], s)):
        with pytest.raises(KernelError):
            K().gemm_f32_parts(*args)
