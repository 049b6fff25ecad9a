"""Which 32-bit attention a step takes (csrc/kernels.py, attention_tiles_pay): the quicker of the two where they were measured (us, one B200,
sequences of equal lengths, query heads over kv heads of a size), and steps of unequal sequences."""
import pytest

from gogguf_b200.csrc.kernels import attention_tiles_pay

# nq, nkv, d, sequences, new tokens, cached positions, a row at a time, in tiles
MEASURED = [
    (16, 8, 128, 1, 16, 0, 5.1, 11.8), (16, 8, 128, 1, 16, 4000, 191.4, 933.5), (16, 8, 128, 1, 32, 900, 69.5, 226.8),
    (16, 8, 128, 1, 64, 6100, 683.0, 1426.7), (16, 8, 128, 1, 128, 900, 225.1, 264.2), (16, 8, 128, 1, 333, 0, 130.9, 105.5),
    (16, 8, 128, 1, 333, 4000, 2299.4, 1306.8), (16, 8, 128, 8, 16, 0, 16.9, 13.5), (16, 8, 128, 8, 16, 900, 214.4, 251.2),
    (16, 8, 128, 3, 64, 0, 30.3, 21.6), (16, 8, 128, 3, 64, 2000, 666.1, 556.0), (16, 8, 128, 8, 64, 900, 830.5, 306.5),
    (16, 8, 64, 1, 16, 900, 48.7, 147.6), (16, 8, 64, 1, 64, 900, 115.5, 158.2), (16, 8, 64, 1, 128, 0, 30.2, 24.4),
    (16, 8, 64, 1, 128, 900, 225.1, 184.9), (16, 8, 64, 1, 333, 900, 620.3, 254.3), (16, 8, 64, 3, 64, 200, 96.6, 54.3),
    (15, 5, 120, 1, 32, 0, 7.7, 12.8), (15, 5, 120, 1, 128, 6100, 1242.2, 1751.8), (15, 5, 120, 1, 333, 900, 582.9, 396.9),
    (15, 5, 120, 8, 16, 900, 198.1, 265.3), (15, 5, 120, 8, 64, 200, 230.0, 97.2),
]


@pytest.mark.parametrize("nq,nkv,d,B,new,cached,rows,tiles", MEASURED)
def test_the_quicker_one(nq, nkv, d, B, new, cached, rows, tiles):
    assert attention_tiles_pay([(cached, new)] * B, nq, nkv, d, d) == (tiles < rows)


def test_unequal_sequences():
    prompt, decode = (0, 450), [(3000, 1)] * 8
    assert attention_tiles_pay([prompt], 16, 8, 128, 128)
    assert not attention_tiles_pay([prompt] + decode, 16, 8, 128, 128)       # a decode row's keys are one chain there
    assert attention_tiles_pay([prompt] + [(40, 1)] * 8, 16, 8, 128, 128)
    assert not attention_tiles_pay([(0, 40)] * 2 + [(600, 1)] * 6, 16, 8, 128, 128)      # under 16 tokens a sequence
    assert not attention_tiles_pay([], 16, 8, 128, 128)                       # lengths that are not known


@pytest.mark.parametrize("bound", [dict(window=256), dict(chunk=256)])
def test_a_bound_on_what_a_token_sees(bound):
    assert attention_tiles_pay([(6100, 333)], 16, 8, 128, 128, **bound)
    assert not attention_tiles_pay([(6100, 16)], 16, 8, 128, 128, **bound)
    assert attention_tiles_pay([(0, 333)], 16, 8, 128, 128, **bound) and not attention_tiles_pay([(0, 16)], 16, 8, 128, 128, **bound)
