"""The strip aligner's blocks fit the device at every length and score the
entry points take: on the CPU by the sizes themselves
(tests/strip_geometry_driver.cpp), on the GPU by whole denoisings of reads
close to the length limit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import dada2_b200 as D
from dada2_b200 import synth
from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_strip_blocks_fit_at_every_length(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path / "strip_geometry_driver")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "dada2-rs_b200", "csrc"), "-I", inc,
                    os.path.join(ROOT, "tests", "strip_geometry_driver.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def sample(seed, length, spread, reads, copies):
    """One variant per entry of ``reads``, ``length - spread`` to ``length``
    bases, and ``copies`` near copies of each, with substitutions and with
    bases dropped from or doubled in homopolymer runs."""
    rng = np.random.default_rng(seed)
    rows, counts = [], []
    for n in reads:
        base = rng.integers(0, 4, length - int(rng.integers(0, spread + 1)))
        rows.append(base)
        counts.append(n)
        for _ in range(copies):
            s = base.copy()
            for p in rng.choice(len(s), 2, replace=False):
                s[p] = (s[p] + rng.integers(1, 4)) % 4
            runs = np.nonzero((s[2:] == s[1:-1]) & (s[1:-1] == s[:-2]))[0] + 1
            p = int(rng.choice(runs))
            s = np.delete(s, p) if rng.random() < 0.5 else np.insert(s, p, s[p])
            rows.append(s[:length])
            counts.append(2)
    seqs = ["".join("ACGT"[x] for x in r) for r in rows]
    quals = [rng.integers(30, 39, len(r)).astype(np.uint32) * n for r, n in zip(rows, counts)]
    return seqs, np.array(counts, np.uint32), quals


def same(got, want):
    assert got["nclust"] == want["nclust"]
    assert np.array_equal(got["map"], want["map"])
    assert got["pvals"].tobytes() == want["pvals"].tobytes()
    for g, w in zip(got["clusters"], want["clusters"]):
        assert np.array_equal(g["members"], w["members"])
        assert np.array_equal(g["hammings"], w["hammings"])
        assert g["lambdas"].tobytes() == w["lambdas"].tobytes()
    for k in ("cmp_scanned", "screened", "aligned", "stored", "gapless", "vectorized", "homo", "endsfree"):
        assert got["counters"][k] == want["counters"][k], k


def denoise(smp, ncol=41, **align):
    seqs, reads, quals = smp
    err = synth.error_matrix(ncol)
    got = D.dada_uniques(seqs, reads, err, ncol, D.DadaParams(align=D.AlignParams(**align), transitions=True),
                         quals=quals)
    want = O.dada(seqs, reads, err, ncol, O.DadaParams(align=O.AlignParams(**align), nthreads=8, transitions=True),
                  quals=quals)
    same(got, want)
    assert np.array_equal(got["transitions"], want["transitions"])
    return want


@pytest.mark.gpu
@pytest.mark.parametrize("length,ncol", [(9240, 41), (9520, 41), (9990, 94)])
def test_longest_reads_match_oracle(length, ncol):
    """Reads the strip aligner takes at mismatch -1 up to 9,990 bases."""
    want = denoise(sample(length, length, 40, (3000, 2000, 400), 5), ncol, mismatch=-1, band=32, homo_gap_p=-1)
    assert want["nclust"] >= 3 and want["counters"]["homo"] > 0
