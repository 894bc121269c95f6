"""Runs of a resident batch of one sample follow one another on two streams: the
next run clears the bounds that the last run's direct calls wrote."""
import numpy as np
import pytest

import dada2_b200 as D
from dada2_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_single_sample_runs_repeat_identically():
    w = synth.small_illumina(64, nvariants=7, nreads=1500, L=110)
    s = w.samples[0]
    want = O.dada(s.seqs, s.abund, w.err, w.ncol, O.DadaParams(nthreads=4), quals=s.quals)
    with D.ResidentBatch([s], w.err, w.ncol, D.DadaParams(host_threads=2)) as rb:
        for _ in range(25):
            got = rb.run()[0]
            assert got["nclust"] == want["nclust"] > 3
            assert np.array_equal(got["map"], want["map"])
            assert got["pvals"].tobytes() == want["pvals"].tobytes()
            assert got["counters"]["stored"] == want["counters"]["stored"]
