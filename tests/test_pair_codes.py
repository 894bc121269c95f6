"""align_pairs with codes other than 1..4, and with the forms that the strip
aligner replaced (a pair with a single base keeps a call on them)."""
import numpy as np
import pytest

import dada2_b200 as D
from oracle import oracle as O
from test_strip_aligner import SCORES, check, pair

ONE = (np.array([1], np.uint8), np.array([2], np.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("letters", [b"ACGT", bytes([1, 2, 17, 18]), bytes([3, 5, 9, 15])])
def test_vectorized_rows_hold_the_bytes_given(letters):
    """Alignments are defined for codes up to 15; rows hold any byte as it came."""
    lut = np.frombuffer(b"?" + letters, np.uint8)
    rng = np.random.default_rng(len(letters) + letters[3])
    pairs = [tuple(lut[x] for x in pair(rng, 120, 120 - t)) for t in range(12)]
    got = D.align_pairs(D.ALIGN_VECTORIZED, pairs, D.AlignParams(band=16))
    for (a, b), (g0, g1) in zip(pairs, got):
        assert np.array_equal(g0[g0 != ord("-")], a) and np.array_equal(g1[g1 != ord("-")], b)
        if max(letters) <= 15:
            w0, w1 = O.align(O.ALIGN_VECTORIZED, a, b, band=16)
            assert np.array_equal(g0, w0) and np.array_equal(g1, w1)


@pytest.mark.gpu
@pytest.mark.parametrize("band,length", [(1, 31), (8, 64), (16, 250), (32, 300), (60, 250), (140, 400), (-1, 90), (32, 1450)])
def test_replaced_forms_match_oracle(band, length):
    """Register, byte-matrix and row-major forms, one pair per warp."""
    rng = np.random.default_rng(31 * length + band)
    pairs = []
    for t in range(16):
        a, b = pair(rng, length, length - (t % 4) * min(9, length // 5), alphabet=2 + t % 3)
        pairs.append((b, a) if t % 2 else (a, b))
    pairs.append(ONE)
    for k, (m, x, g) in enumerate(SCORES):
        check(D.ALIGN_VECTORIZED, pairs, band, m, x, g, g)
        check(D.ALIGN_ENDSFREE, pairs, band, m, x, g, g)
        check(D.ALIGN_HOMO, pairs, band, m, x, g, (-1, 0, -3, -1)[k])
