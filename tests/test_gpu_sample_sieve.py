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
