"""Direct compare calls (late clusters: comps stored and posted by the
alignment kernel) against the oracle, around the number of pairs they post."""
import numpy as np
import pytest

import dada2_b200 as D
from dada2_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

POST_MAX = 4096  # pairs a direct call posts; it is made again with the store kernel past that


def sample(seed, small, large, L=100):
    """Three unrelated variants: the most abundant, one with ``small`` uniques
    (its call is followed by a direct one) and one with ``large``."""
    rng = np.random.default_rng(seed)
    a, b, c = (rng.integers(0, 4, L) for _ in range(3))
    rows, reads = [a, b, c], [30000, 20000, 4000]

    def copies(base, n):
        seen = set()
        while len(seen) < n:
            s = base.copy()
            for p in rng.choice(L, 2, replace=False):
                s[p] = (s[p] + rng.integers(1, 4)) % 4
            seen.add(s.tobytes())
        return [np.frombuffer(k, base.dtype) for k in sorted(seen)]

    for base, n in ((b, small), (c, large)):
        rows += copies(base, n)
        reads += [2] * n
    seqs = ["".join("ACGT"[x] for x in r) for r in rows]
    return seqs, np.array(reads, np.uint32), [np.full(L, 38 * r, np.uint32) for r in reads]


@pytest.mark.parametrize("large", [200, POST_MAX - 2, POST_MAX - 1, POST_MAX + 300])
def test_direct_calls_match_oracle(large):
    """The third cluster's call queues its center and ``large`` pairs."""
    seqs, reads, quals = sample(large, 30, large)
    err = synth.error_matrix(41)
    got = D.dada_uniques(seqs, reads, err, 41, D.DadaParams(), quals=quals)
    want = O.dada(seqs, reads, err, 41, O.DadaParams(nthreads=8), quals=quals)
    assert got["nclust"] == want["nclust"] >= 3
    assert np.array_equal(got["map"], want["map"])
    assert got["pvals"].tobytes() == want["pvals"].tobytes()
    for g, w in zip(got["clusters"], want["clusters"]):
        assert np.array_equal(g["members"], w["members"])
        assert g["lambdas"].tobytes() == w["lambdas"].tobytes()
    for k in ("cmp_scanned", "screened", "aligned", "stored", "gapless", "vectorized"):
        assert got["counters"][k] == want["counters"][k], k
