"""The top-k kernel's sieve (csrc/sampling.cu): around the largest k it takes, rows it cannot thin out, ties and short
slices, against the host chain; and the batch's uniform numbers against the single ones."""
import numpy as np
import pytest
import torch


def test_uniforms_of_a_batch():
    from gogguf_b200.sampling.sampler import _uniforms, uniform01
    for n in (0, 1, 3, 4, 70):
        streams, steps = [5 - i for i in range(n)], [(1 << 62) + 977 * i for i in range(n)]
        for seed in (0, 12345, -1, 1 << 70):
            assert _uniforms(seed, streams, steps) == [uniform01(seed, s, k) for s, k in zip(streams, steps)]


@pytest.mark.gpu
@pytest.mark.parametrize("V", [40, 8192, 8200, 30011])
@pytest.mark.parametrize("top_k", [1, 20, 64, 65, 511, 512, 513])
def test_rows_through_the_sieve(V, top_k):
    from gogguf_b200.sampling.sampler import Sampler, SamplerConfig, sample_host, uniform01
    g = torch.Generator().manual_seed(V + top_k)
    normal = torch.randn(V, generator=g) * 3
    ids = torch.arange(V)
    rows = [normal, normal.sort().values, torch.zeros(V), (normal * 2).round(),
            normal + 40.0 * (ids % 256 < 125),          # some 4,000 large values in 500 groups: more than the sieve has room for
            normal + 40.0 * (ids % 256 < 2), torch.where(ids % 3 == 0, normal, torch.tensor(-float("inf")))]
    cfg = SamplerConfig(temp=0.7, top_k=top_k, top_p=0.9, seed=5)
    logits = torch.stack(rows)
    for step in range(3):
        got = Sampler(cfg).sample(logits.cuda(), list(range(len(rows))), [step] * len(rows))
        want = [sample_host(r.numpy().astype(np.float32), cfg, uniform01(5, i, step)) for i, r in enumerate(rows)]
        assert got == want


@pytest.mark.gpu
@pytest.mark.parametrize("V", [64, 8191, 16388])
@pytest.mark.parametrize("temp,top_k", [(0.75, 20), (1.0, 20), (0.875, 24), (1.75, 25), (2.0 ** 20, 20), (2.0 ** -20, 7), (0.625, 64)])
def test_sieve_before_the_division(V, temp, top_k):
    """The sieve runs on undivided logits: values a step apart that the division makes equal (the lower id wins), quotients that
    vanish, many zeros, infinities (temperatures that
    32 bits hold, as the host's 64 do; no top-p: the host orders equal probabilities by id); more rows than one launch carries numbers for."""
    from gogguf_b200.sampling.sampler import Sampler, SamplerConfig, sample_host, uniform01
    g = torch.Generator().manual_seed(V + top_k)
    steps_apart = torch.tensor(5.0).view(torch.int32) + torch.randint(0, 12, (V,), generator=g, dtype=torch.int32)
    normal = torch.randn(V, generator=g)
    ids = torch.arange(V)
    rows = [normal, steps_apart.view(torch.float32), -steps_apart.view(torch.float32), normal.abs() * 1e-38,
            torch.where(ids % 2 == 0, torch.tensor(0.0), normal), torch.where(ids < V - top_k // 2, -normal.abs(), normal.abs()),
            torch.where(ids % 5 == 0, normal, torch.tensor(-float("inf")))]
    cfg = SamplerConfig(temp=temp, top_k=top_k, seed=-3)
    logits = torch.stack(rows * 40)
    n = len(logits)
    got = Sampler(cfg).sample(logits.cuda(), [-5 + i for i in range(n)], [3] * n)
    want = [sample_host(logits[i].numpy(), cfg, uniform01(-3, i - 5, 3)) for i in range(n)]
    assert n > 256 and got == want
