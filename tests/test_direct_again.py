"""A direct compare call that queues more pairs than it posts is made again with
the store kernel: the call counts once in the library's figures, its launches
as often as they ran."""
import pytest

import dada2_b200 as D
from dada2_b200 import synth
from test_direct_calls import POST_MAX, sample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,again", [(200, 0), (POST_MAX + 300, 1)])
def test_a_call_made_again_counts_once(large, again):
    seqs, reads, quals = sample(large, 30, large)
    err = synth.error_matrix(41)
    D.stats_reset()
    r = D.dada_uniques(seqs, reads, err, 41, D.DadaParams(), quals=quals)
    st = D.stats_read()
    assert st["rounds"] == r["counters"]["compare_calls"] == len(D.stats_latencies())
    assert st["compares"] == r["counters"]["cmp_scanned"]
    assert st["screened"] == r["counters"]["screened"]
    assert st["launches"]["screen"] == st["rounds"] + again
