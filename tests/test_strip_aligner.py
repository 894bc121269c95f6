"""The strip aligner (one DP for the vectorized and the row-major aligners).

It rests on the two choosing the same moves for end gap 0 and sequences of two
or more bases; on the GPU its alignments are compared byte for byte with the
oracle's at the edges of its strips (bands of 62 C diagonals), of its pointer
words (lengths around multiples of their rows) and of its shared-memory form.
"""
import numpy as np
import pytest

import dada2_b200 as D
from oracle import oracle as O

SCORES = [(5, -4, -8), (1, -1, -2), (2, -3, -1), (5, -4, 0)]


def pair(rng, l1, l2, alphabet=4):
    """A sequence of l1 bases and a mutated copy brought to l2 bases."""
    a = rng.integers(1, alphabet + 1, l1)
    b = list(a)
    for _ in range(int(rng.integers(0, 7))):
        p, op = int(rng.integers(0, len(b))), int(rng.integers(0, 3))
        if op == 0:
            b[p] = int(rng.integers(1, alphabet + 1))
        elif op == 1:
            b[p:p] = [b[p]] * int(rng.integers(1, 5))
        elif len(b) > 5:
            del b[p:p + int(rng.integers(1, 4))]
    cut = int(rng.integers(0, max(1, len(b) - l2 + 1)))
    b = b[cut:cut + l2] if len(b) >= l2 else b + list(rng.integers(1, alphabet + 1, l2 - len(b)))
    return a.astype(np.uint8), np.array(b, np.uint8)


@pytest.mark.parametrize("band", [1, 2, 5, 15, 16, 17, 32, 33, 100, -1])
def test_vectorized_and_row_major_aligners_choose_the_same_moves(band):
    rng = np.random.default_rng(4000 + band)
    for t in range(400):
        l1 = int(rng.integers(2, 90))
        l2 = l1 if t % 3 == 0 else max(2, l1 + int(rng.integers(-40, 41)))
        a, b = pair(rng, l1, l2, alphabet=2 + t % 3)
        if t % 4 == 0:
            b = rng.integers(1, 5, l2).astype(np.uint8)
        m, x, g = SCORES[t % 4]
        v = O.align(O.ALIGN_VECTORIZED, a, b, match=m, mismatch=x, gap=g, homo_gap=g, band=band)
        r = O.align(O.ALIGN_ENDSFREE, a, b, match=m, mismatch=x, gap=g, homo_gap=g, band=band)
        assert np.array_equal(v[0], r[0]) and np.array_equal(v[1], r[1]), (l1, l2, band, m, x, g)


def check(which, pairs, band, m, x, g, hg):
    owhich = {D.ALIGN_VECTORIZED: O.ALIGN_VECTORIZED, D.ALIGN_HOMO: O.ALIGN_HOMO,
              D.ALIGN_ENDSFREE: O.ALIGN_ENDSFREE}[which]
    p = D.AlignParams(band=band, match_score=m, mismatch=x, gap_p=g, homo_gap_p=hg)
    got = D.align_pairs(which, pairs, p)
    for (a, b), (g0, g1) in zip(pairs, got):
        w0, w1 = O.align(owhich, a, b, match=m, mismatch=x, gap=g, homo_gap=hg, band=band)
        assert np.array_equal(g0, w0) and np.array_equal(g1, w1), (which, len(a), len(b), band, m, x, g, hg)


@pytest.mark.gpu
@pytest.mark.parametrize("width", [3, 33, 62, 63, 64, 124, 125, 126, 128, 186, 187, 192, 248, 249, 256])
@pytest.mark.parametrize("length", [9, 31, 97, 250, 500, 521])
def test_strip_aligner_matches_oracle(width, length):
    """Bands of ``width`` diagonals in the widest pair, in both orientations."""
    rng = np.random.default_rng(17 * width + length)
    diff = min((width - 1) % 31, length - 2, width - 3)
    band = (width - 1 - diff) // 2
    diff = min(width - 1 - 2 * band, length - 2)
    pairs = []
    for t in range(24):
        l2 = length - (diff if t % 3 == 0 else int(rng.integers(0, diff + 1)))
        a, b = pair(rng, length, l2, alphabet=2 + t % 3)
        pairs.append((b, a) if t % 2 else (a, b))
    for k, (m, x, g) in enumerate(SCORES):
        check(D.ALIGN_VECTORIZED, pairs, band, m, x, g, g)
        check(D.ALIGN_ENDSFREE, pairs, band, m, x, g, g)
        check(D.ALIGN_HOMO, pairs, band, m, x, g, (-1, 0, -3, -1)[k])


@pytest.mark.gpu
@pytest.mark.parametrize("lmax", [2, 3, 1550, 2497, 2498])
def test_strip_aligner_at_its_length_limits(lmax):
    """The shortest pairs, full-length ones and the last length the row-major
    aligners' band marks allow (2,497 bases at mismatch -4), and one past it."""
    rng = np.random.default_rng(lmax)
    pairs = [pair(rng, lmax, max(2, lmax - int(rng.integers(0, 60)))) for _ in range(6)]
    check(D.ALIGN_HOMO, pairs, 32, 5, -4, -8, -1)
    check(D.ALIGN_HOMO, [pair(rng, lmax, max(2, lmax - 61 * (t % 4))) for t in range(8)], 32, 5, -4, -8, -1)
    check(D.ALIGN_ENDSFREE, pairs, 32, 5, -4, -8, -8)
    check(D.ALIGN_VECTORIZED, pairs, 16, 5, -4, -8, -8)
