"""The rule that a pair's plain diagonal alignment beats every other one, shown
without the DP (diagonal_is_best): on the CPU a mirror of it against the
oracle's aligner, on the GPU a compare call against the oracle's."""
import numpy as np
import pytest

import dada2_b200 as D
from dada2_b200 import synth
from oracle import oracle as O


def rule(s, t):
    """diagonal_is_best's answer, by rows instead of words of 32."""
    L, p = len(s), np.nonzero(s != t)[0]
    m = len(p)
    if L < 128 or L > 512 or m > 3:
        return False
    if m == 0:
        return True
    x = {}
    for d in (*range(-5, 0), *range(1, 6)):
        rows = np.arange(max(0, -d), min(L, L - d))
        x[d] = np.zeros(L, bool)
        x[d][rows] = s[rows] != t[rows + d]
        if any(x[d][32 * w:32 * w + 32].sum() < 10 for w in range(L // 32)):
            return False

    def shown(of, lo, hi, k):
        return all(of(side)[max(lo, 0):max(hi + 1, 0)].sum() >= k for side in (1, -1))

    def one(side):
        return x[side]

    def two(side):
        return x[side] & x[2 * side]

    if m == 1:
        return True
    if m == 2:
        return shown(one, 1, p[1] - 1, 1) and shown(one, p[0] + 1, L - 2, 1)
    return (shown(one, p[0] + 1, p[2] - 1, 1) and shown(one, 1, p[1] - 1, 1) and shown(one, p[1] + 1, L - 2, 1) and
            shown(one, 2, p[2] - 2, 2) and shown(one, p[0] + 2, L - 3, 2) and
            shown(two, 2, p[2] - 2, 3) and shown(two, p[0] + 2, L - 3, 3))


def sequence(rng, L):
    """Random bases with periodic stretches at the ends and inside."""
    s = rng.integers(1, 5, L)
    for a in (0, L - 40, int(rng.integers(0, L - 45))):
        if rng.random() < 0.5:
            unit = rng.integers(1, 5, int(rng.integers(1, 6)))
            w = int(rng.integers(3, 40))
            s[a:a + w] = np.resize(unit, w)
    return s.astype(np.uint8)


def copy_of(rng, s):
    """Up to three substitutions, often close together and often to a neighbouring base."""
    L, t = len(s), s.copy()
    w = int(rng.choice([4, 8, 14, 40, L]))
    a = int(rng.choice([0, int(rng.integers(0, L - w + 1)), L - w]))
    for p in a + rng.choice(w, int(rng.integers(1, 4)), replace=False):
        near = int(np.clip(p + rng.choice([-2, -1, 1, 2]), 0, L - 1))
        t[p] = s[near] if rng.random() < 0.5 and s[near] != s[p] else (s[p] - 1 + rng.integers(1, 4)) % 4 + 1
    return t


@pytest.mark.parametrize("seed", range(4))
def test_rule_never_accepts_a_pair_whose_best_alignment_has_gaps(seed):
    rng = np.random.default_rng(900 + seed)
    accepted = gaps = 0
    for _ in range(2500):
        s = sequence(rng, int(rng.integers(128, 300)))
        t = copy_of(rng, s)
        a0, a1 = O.align(O.ALIGN_VECTORIZED, s, t, band=16)
        plain = len(a0) == len(s) and np.array_equal(a0, s) and np.array_equal(a1, t)
        gaps += not plain
        if rule(s, t):
            accepted += 1
            assert plain, (s, t)
    assert accepted > 1000 and gaps > 10


@pytest.mark.gpu
@pytest.mark.parametrize("L", [127, 128, 159, 160, 250, 300, 480, 511, 512, 513])
def test_compare_of_near_copies_matches_oracle(L):
    """One center against near copies, with the gapless shortcut off so that all take the rule or the DP."""
    rng = np.random.default_rng(L)
    s = sequence(rng, L)
    rows = [s] + [copy_of(rng, s) for _ in range(400)]
    # rows with a base left out or doubled go through the DP
    rows += [np.concatenate([s[:p], s[p + 1:], s[:1]]) for p in rng.integers(1, L - 1, 20)]
    reads = np.array([1000] + [1] * (len(rows) - 1), np.uint32)
    quals = [rng.integers(2, 41, L).astype(np.uint8) for _ in rows]
    err = synth.error_matrix(41)
    ctx = D.CompareContext(D.AlignParams(gapless=False), err, 41)
    ctx.upload(rows, reads, quals)
    lam, ham, skipped, counters = ctx.compare(0, 1.0)
    ses = O.Session(rows, reads, quals)
    ses.set_center(0, 0)
    want = ses.compare_map(0, err, 41, O.AlignParams(gapless=False, kdist_cutoff=1.0))
    assert lam.tobytes() == want[0].tobytes()
    assert np.array_equal(ham, want[1]) and np.array_equal(skipped, want[2])
    assert counters["vectorized"] == len(rows)
