"""Compare calls and denoisings that the strip aligner does not take: long reads
with homopolymer gaps (the row-major form, its cooperative mode, and their
direct stores), more than 248 diagonals, pools that span the vectorized
aligner's length limit, and scores past the strip rule. Reads this long leave
room for fewer blocks than the launch would otherwise have."""
import numpy as np
import pytest

import dada2_b200 as D
from dada2_b200 import synth
from oracle import oracle as O
from test_strip_geometry import denoise, sample

pytestmark = pytest.mark.gpu

READS = (3000, 2000, 900, 400)


@pytest.mark.parametrize("length,spread,copies,align,method", [
    (2600, 40, 30, dict(band=32, homo_gap_p=-1), "homo"),  # two lane groups: a block's warps share each pair
    (2600, 40, 12, dict(band=80, homo_gap_p=-1), "homo"),  # four
    (400, 20, 30, dict(band=140, homo_gap_p=-1), "homo"),  # eight: one warp per pair
    (2600, 40, 30, dict(band=12, homo_gap_p=-1), "homo"),  # one
    (400, 20, 30, dict(band=140), "vectorized"),
    (300, 0, 30, dict(band=16, gap_p=-1100, homo_gap_p=-1100), "vectorized"),
    (3560, 120, 15, dict(band=16), "endsfree"),  # vectorized and row-major pairs in one call
    (4000, 40, 110, dict(band=16), "endsfree"),
    (3400, 40, 150, dict(band=16), "vectorized"),  # the strip aligner, three blocks per SM
])
def test_denoising_matches_oracle(length, spread, copies, align, method):
    want = denoise(sample(length + copies, length, spread, READS, copies), **align)
    assert want["nclust"] >= 4 and want["counters"][method] > 0
    if length == 3560:
        assert want["counters"]["vectorized"] > 0


@pytest.mark.parametrize("length,copies,align", [
    (2600, 30, dict(band=32, homo_gap_p=-1)),
    (2600, 330, dict(band=20, homo_gap_p=-1)),  # more pairs than the cooperative mode takes
    (4000, 110, dict(band=16)),
    (3400, 150, dict(band=16)),
])
def test_compare_call_matches_oracle(length, copies, align):
    seqs, reads, quals = sample(length + 1, length, 40, READS, copies)
    rows = [np.array(["ACGT".index(c) + 1 for c in s], np.uint8) for s in seqs]
    q = [(a // n).astype(np.uint8) for a, n in zip(quals, reads)]
    err = synth.error_matrix(41)
    with D.CompareContext(D.AlignParams(**align), err, 41) as ctx:
        ctx.upload(rows, reads, q)
        lam, ham, skipped, counters = ctx.compare(0, 1.0, greedy=False)
    ses = O.Session(rows, reads, q)
    ses.set_center(0, 0)
    want = ses.compare_map(0, err, 41, O.AlignParams(kdist_cutoff=1.0, **align), greedy=False, nthreads=8)
    assert lam.tobytes() == want[0].tobytes()
    assert np.array_equal(ham, want[1]) and np.array_equal(skipped, want[2])
    assert counters["aligned"] == len(rows)
