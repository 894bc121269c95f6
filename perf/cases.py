"""The work a user has this framework do, as timed cases through its public entry points.

A case is a dict of plain values; ``kind`` names the entry point:

* ``map``     one compare call (``CompareContext.compare``) over resident uniques;
* ``store``   a sample's first compare call and a later cluster's one with their
              stores (``CompareContext.b_compare_parallel``);
* ``dada``    one sample denoised from host buffers (``dada_uniques``);
* ``batch``   resident samples denoised together (``ResidentBatch.run``);
* ``learn``   the error model learned from samples (``learn_errors``);
* ``service`` requests of mixed lengths through a resident ``DenoiseService``.

The inputs are amplicon reads simulated on the device from the seed: variants
of uniform-random bases, reads drawn by an abundance law, substitutions by the
16 x quality error model, dereplicated with per-position Phred sums. Long reads
also carry indels in homopolymer runs and have binned qualities.
"""
from __future__ import annotations

import os
import sys
from types import SimpleNamespace

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dada2-rs_b200"))

import dada2_b200 as D  # noqa: E402

KMER = 5
CUTOFF = 0.42
LETTERS = np.frombuffer(b"?ACGT", np.uint8)
RESULT_KEYS = ("cl_reads", "cl_birth_type", "cl_birth_from", "cl_birth_pval", "cl_birth_fold", "cl_birth_e",
               "cl_birth_hamming", "cl_seq", "mem_raw", "mem_hamming", "mem_lambda", "mem_pval", "map", "pvals")


def listed():
    return [
        # the smallest drop-in call: a late cluster of a small sample against every unique
        {"name": "map_1k_250", "kind": "map", "uniques": 1000, "length": 250, "variants": 20, "late": True},
        # one call over a pooled V4 run, the most uniques a single call meets
        {"name": "map_400k_150", "kind": "map", "uniques": 400000, "length": 150, "variants": 3000, "late": True},
        # PacBio full-length 16S: cluster 0's call aligns every unique (band 32, homopolymer gaps)
        {"name": "map_long_5k", "kind": "map", "uniques": 5000, "length": 1550, "spread": 150, "variants": 60,
         "long": True},
        # the first and a later compare call of a large Illumina sample, with their stores
        {"name": "store_30k_250", "kind": "store", "uniques": 30000, "length": 250, "variants": 200},
        # a shallow V4 sample with lengths a few bases apart, where a call's fixed costs count
        {"name": "dada_500_153", "kind": "dada", "uniques": 500, "length": 153, "spread": 3, "variants": 12},
        # the plain single Illumina sample (20 variants, 20,000 reads)
        {"name": "dada_3k_250", "kind": "dada", "uniques": 3000, "length": 250, "variants": 20},
        # a deep sample with many variants and the transition counts of the final pass
        {"name": "dada_16k_250", "kind": "dada", "uniques": 16000, "length": 250, "variants": 400,
         "transitions": True},
        # a PacBio full-length 16S sample end to end
        {"name": "dada_long_5k", "kind": "dada", "uniques": 5000, "length": 1550, "spread": 150, "variants": 60,
         "long": True},
        # 200 samples pooled into one, the largest single denoising
        {"name": "dada_pooled_400k", "kind": "dada", "uniques": 400000, "length": 150, "variants": 3000,
         "pooled": True},
        # a sequencing run's samples (forward and reverse lengths) denoised together
        {"name": "batch_40", "kind": "batch", "samples": 40, "umin": 500, "umax": 30000, "length": 250,
         "length2": 220, "vmin": 50, "vmax": 400},
        # the error model of a run, from six of its samples
        {"name": "learn_6", "kind": "learn", "samples": 6, "umin": 500, "umax": 12000, "length": 250,
         "length2": 220, "vmin": 50, "vmax": 200},
        # requests of three read lengths served by one resident service
        {"name": "service_16", "kind": "service", "samples": 16, "umin": 1000, "umax": 20000, "length": 250,
         "length2": 150, "vmin": 50, "vmax": 200, "longs": 1},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["map", "map", "store", "dada", "dada", "dada", "batch", "learn", "service"])
    case = {"kind": kind, "length": rng.randint(120, 300)}
    if kind in ("map", "store", "dada"):
        long = kind != "store" and rng.random() < 0.3
        top = 5000 if long else {"map": 400000, "store": 60000, "dada": 30000}[kind]
        n = log(500, top)
        case.update(uniques=n, variants=log(10, 60 if long else 400) + n // 200, long=long,
                    spread=rng.randint(20, 150) if long else rng.choice([0, 0, 3, 7, 12]))
        if long:
            case["length"] = rng.randint(1200, 1550)
        if kind == "map":
            case["late"] = rng.random() < 0.5
        if kind == "dada":
            case["transitions"] = rng.random() < 0.5
    else:
        case.update(samples=rng.randint(2, 6) if kind == "learn" else rng.randint(4, 16 if kind == "service" else 40),
                    umin=500, umax=log(2000, 12000 if kind == "learn" else 30000), length2=rng.randint(120, 300),
                    vmin=10, vmax=rng.randint(40, 400))
        if kind == "service":
            case["longs"] = rng.choice([0, 0, 1])
    return case


# ---- inputs -------------------------------------------------------------------


def error_model(ncol: int, floor: float = 0.0) -> np.ndarray:
    """16 x ncol: row 4 * ref + query, column quality; error rate 10^(-Q/10),
    transitions twice as likely as transversions."""
    e = np.maximum(10.0 ** (-np.arange(ncol) / 10.0), floor)
    share = np.array([[0, 1, 2, 1], [1, 0, 1, 2], [2, 1, 0, 1], [1, 2, 1, 0]]) / 4.0
    m = np.clip(share[:, :, None] * e, 1e-7, 0.25)
    m[range(4), range(4)] = 0.0
    m[range(4), range(4)] = 1.0 - m.sum(axis=1)
    return np.ascontiguousarray(m.reshape(16, ncol))


def model_of(case: dict):
    return (error_model(94, 1e-3), 94) if case.get("long") else (error_model(42), 42)


def params_of(case: dict) -> D.DadaParams:
    align = D.AlignParams(band=32, homo_gap_p=-1) if case.get("long") else D.AlignParams(band=16)
    return D.DadaParams(align=align, transitions=bool(case.get("transitions")))


def substitute(codes, quals, gen, model):
    """Substitutions at the quality's rate, the new base by the model's row."""
    cum = torch.from_numpy(model.reshape(4, 4, -1).cumsum(axis=1)).to(codes.device, torch.float32)
    u = torch.rand(codes.shape, generator=gen, device=codes.device)
    ref, q = codes.long() - 1, quals.long()
    new = torch.ones_like(codes)
    for b in range(3):
        new += (u > cum[ref.clamp(min=0), b, q]).to(codes.dtype)
    return torch.where(codes > 0, new, codes)


def dereplicate(codes, quals, key, gen, pooled: bool, uniques: int):
    """``uniques`` distinct rows (those read once are thinned at random) with
    counts and quality sums, by (-count, row), or in first-seen order for a
    pooled sample. ``key`` is the same for equal rows."""
    dev, width = codes.device, codes.shape[1]
    _, inverse, count = torch.unique(key, return_inverse=True, return_counts=True)
    n, index = count.numel(), torch.arange(key.numel(), device=dev)
    first = torch.full((n,), key.numel(), device=dev).scatter_reduce_(0, inverse, index, "amin")
    sums = torch.zeros((n, width), dtype=torch.int32, device=dev)
    for part, inv in zip(quals.split(200000), inverse.split(200000)):
        sums.index_add_(0, inv, part.int())
    rank = torch.rand(n, generator=gen, device=dev) + (count > 1)
    keep = rank.argsort(descending=True)[:uniques].sort().values
    first, count, sums, n = first[keep], count[keep], sums[keep], uniques
    rows = codes[first]
    if pooled:
        order = first.argsort()
    else:
        order = torch.arange(n, device=dev)
        for lo in reversed(range(0, width, 20)):  # twenty codes of three bits to a word
            part = rows[:, lo:lo + 20].long()
            word = (part << (3 * torch.arange(19, 19 - part.shape[1], -1, device=dev))).sum(1)
            order = order[word[order].argsort(stable=True)]
        order = order[(-count)[order].argsort(stable=True)]
    return rows[order].cpu().numpy(), count[order].cpu().numpy().astype(np.uint32), sums[order].cpu().numpy()


def simulate(seed: int, uniques: int, length: int, variants: int, spread: int = 0, long: bool = False,
             pooled: bool = False):
    """One sample: code rows (1..4, 0 past the end), counts and quality sums."""
    dev = torch.device("cuda")
    gen = torch.Generator(dev).manual_seed(seed)
    lens = length - torch.randint(0, spread + 1, (variants,), generator=gen, device=dev)
    base = torch.randint(1, 5, (variants, length), generator=gen, device=dev, dtype=torch.int8)
    base[torch.arange(length, device=dev)[None, :] >= lens[:, None]] = 0
    if pooled:  # log-normal abundances (sigma 2)
        weight = torch.exp(2.0 * torch.randn(variants, generator=gen, device=dev, dtype=torch.float64))
    else:
        weight = torch.arange(1, variants + 1, device=dev, dtype=torch.float64) ** (-1.0 if long else -1.5)
    if long:
        model, width = error_model(94, 2e-3), length + 65
        same = base[:, 1:] == base[:, :-1]
        run = torch.zeros_like(base, dtype=torch.bool)
        run3 = same[:, 1:] & same[:, :-1] & (base[:, 2:] > 0)
        for s in range(3):
            run[:, s:length - 2 + s] |= run3
        bins = torch.tensor([40, 50, 60, 70, 80, 93], device=dev, dtype=torch.int8)
    else:
        model, width = error_model(42), length
        profile = torch.linspace(38.0, 25.0, length, device=dev)
    mix = torch.randint(-2 ** 62, 2 ** 62, (width,), generator=gen, device=dev) | 1
    codes, quals, keys, seen = [], [], [], 0
    # more reads until they hold the uniques; at first as many as if few repeated
    reads = step = int(uniques / (1.0 if long else min(0.11 * (length / 150.0) ** 1.3, 0.9)))
    while seen < uniques:
        pick = torch.multinomial(weight, step, replacement=True, generator=gen)
        for p in pick.split(4000 if long else 500000):
            if long:
                hit = (torch.rand((len(p), length), generator=gen, device=dev) < 5e-3) & run[p]
                twice = torch.rand((len(p), length), generator=gen, device=dev) < 0.5
                copies = (base[p] > 0).long() + hit * (2 * twice.long() - 1)  # a base of a run dropped or doubled
                end = copies.cumsum(1)
                c = torch.zeros((len(p), width), dtype=torch.int8, device=dev)
                for k in range(2):
                    at = torch.where(copies > k, end - copies + k, width - 1)
                    c.scatter_(1, at.clamp(max=width - 1), base[p])
                c[:, width - 1:] = 0
                q = bins[torch.randint(0, 6, c.shape, generator=gen, device=dev)] * (c > 0)
                c = substitute(c, q.clamp(max=40), gen, model)
            else:
                c = base[p]
                noise = torch.randn((len(p), length), generator=gen, device=dev)
                q = (profile + 2.0 * noise).round_().clamp_(2, 41).to(torch.int8) * (c > 0)
                c = substitute(c, q, gen, model)
            codes.append(c)
            quals.append(q)
            keys += [(part.long() * mix).sum(1) for part in c.split(200000)]
        seen = torch.unique(torch.cat(keys)).numel()
        step = reads // 2
    return dereplicate(torch.cat(codes), torch.cat(quals), torch.cat(keys), gen, pooled, uniques)


def sample_of(seed: int, **shape):
    """A sample as the entry points take it: sequences, counts, quality sums."""
    rows, count, sums = simulate(seed, **shape)
    lens = (rows > 0).sum(axis=1)
    text = LETTERS[rows].tobytes()
    w = rows.shape[1]
    sums = sums.astype(np.uint32)
    return SimpleNamespace(seqs=[text[i * w:i * w + n] for i, n in enumerate(lens)], abund=count,
                           quals=[sums[i, :n] for i, n in enumerate(lens)])


def shape_of(case: dict) -> dict:
    return {k: case.get(k, 0) for k in ("uniques", "length", "variants", "spread", "long", "pooled")}


def shapes_of(case: dict) -> list:
    """The samples of a batch: uniques log-uniform, two lengths in turn; the
    sizes are the case's, the reads the seed's."""
    rng = np.random.default_rng(1001)
    shapes = []
    for i in range(case["samples"]):
        lo, hi = case["umin"], case["umax"]
        n = int(lo * (hi / lo) ** rng.random())
        shapes.append({"uniques": n, "length": case["length2"] if i % 2 else case["length"],
                       "variants": int(rng.integers(case["vmin"], case["vmax"] + 1))})
    for i in range(case.get("longs", 0)):  # long reads under the Illumina model: 1,450 nt
        shapes[i * 5 + 2].update(uniques=2000, length=1450)
    return shapes


def encoded(case: dict, seed: int):
    """Codes, counts and rounded mean qualities for a compare context."""
    rows, count, sums = simulate(seed, **shape_of(case))
    mean = np.floor(sums / count[:, None].astype(np.float64) + 0.5).astype(np.uint8)
    return rows.astype(np.uint8), (rows > 0).sum(axis=1), count, mean


def late_center(rows, lens, count) -> int:
    """A later cluster's center: the most abundant unique that shares no more
    with the first than unrelated sequences do."""
    near = (rows[:, :100] == rows[0, :100]).mean(axis=1)
    return int(np.argmax(np.where(near < 0.5, count, 0)))


def prepare(case: dict, seed: int):
    kind = case["kind"]
    err, ncol = model_of(case)
    state = {"kind": kind, "err": err, "ncol": ncol, "params": params_of(case), "late": bool(case.get("late"))}
    if kind in ("map", "store"):
        rows, lens, count, mean = encoded(case, seed)
        ctx = D.CompareContext(state["params"].align, err, ncol)
        ctx.upload([r[:n] for r, n in zip(rows, lens)], count, [q[:n] for q, n in zip(mean, lens)])
        state.update(ctx=ctx, center=late_center(rows, lens, count))
    elif kind == "dada":
        state["room"] = (2 * case["variants"] + 32, case["length"] + 64)
        s = sample_of(seed, **shape_of(case))
        state["packed"] = D.pack_sample(s.seqs, s.abund, s.quals)
    else:
        shapes = shapes_of(case)
        samples = [sample_of(seed * 100 + i, **shape) for i, shape in enumerate(shapes)]
        state["room"] = (sum(2 * s["variants"] + 32 for s in shapes), max(s["length"] for s in shapes))
        if kind == "learn":
            state["samples"] = samples
        elif kind == "batch":
            state["batch"] = D.ResidentBatch(samples, err, ncol, state["params"])
        else:
            state["service"] = D.DenoiseService(err, ncol, state["params"])
            state["packed"] = [D.pack_sample(s.seqs, s.abund, s.quals) for s in samples]
    return state


# ---- one pass -----------------------------------------------------------------


def padded(a, size: int):
    return np.concatenate([a, np.zeros(size - len(a), a.dtype)])


def tables(results, clusters: int, length: int) -> dict:
    """The result tables of one or more samples, one array per table; those of
    the clusters end in zeros up to a size that holds every seed's."""
    out = {k: np.concatenate([r[k] for r in results]) for k in RESULT_KEYS}
    for k, a in out.items():
        if k.startswith("cl_"):
            out[k] = padded(a, clusters * length if k == "cl_seq" else clusters)
    if "transitions" in results[0]:
        out["transitions"] = np.concatenate([r["transitions"].reshape(-1) for r in results])
    return out


def run(state):
    kind = state["kind"]
    if kind == "map":
        if state["late"]:
            return state["ctx"].compare(state["center"], CUTOFF)
        return state["ctx"].compare(0, 1.0)
    if kind == "store":
        ctx = state["ctx"]
        ctx.reset_e_minmax()
        calls = [ctx.b_compare_parallel(0, 0, 1.0), ctx.b_compare_parallel(state["center"], 1, CUTOFF)]
        for call in calls:
            for k in ("index", "lambda", "hamming"):
                call[k] = padded(call[k], ctx.n)
        return {"first": calls[0], "later": calls[1], "e_minmax": ctx.e_minmax()}
    if kind == "dada":
        return tables([D.dada_uniques(None, None, state["err"], state["ncol"], state["params"],
                                      packed=state["packed"])], *state["room"])
    if kind == "batch":
        return tables(state["batch"].run(), *state["room"])
    if kind == "learn":
        return D.learn_errors(state["samples"], state["params"])
    service = state["service"]
    tickets = [service.submit(packed=p) for p in state["packed"]]
    return tables([service.wait(t)[0] for t in tickets], *state["room"])


def work(case: dict) -> dict:
    """The inputs read once, the tables written once, and per compare call the
    shared k-mers of every unique, per aligned pair its band's cells (five
    operations each) and the lambda product. Every unique is aligned about
    twice: against the first center and against its own."""
    kind = case["kind"]
    if kind in ("map", "dada", "store"):
        shapes = [shape_of(case)]
    else:
        shapes = shapes_of(case)
    band = 32 if case.get("long") else 16
    size = ops = 0
    for s in shapes:
        n, length = s["uniques"], s["length"]
        calls, pairs = s["variants"], 2 * n
        if kind == "map":
            calls, pairs = 1, n // 10 if case.get("late") else n
        elif kind == "store":
            calls = 2
        elif kind == "learn":
            pairs = 3 * n
        per = 2 * length + 13 if kind in ("map", "store") else 5 * length + 40
        size += n * per
        ops += calls * n * (length - KMER + 1) + pairs * (length * (2 * band + 1) * 5 + length)
    return {"bytes": size, "flops": ops}


# ---- what a compare call returns, in 64 bits ------------------------------------


def kmer_counts(rows, lens):
    n, width = rows.shape
    windows = width - KMER + 1
    code = torch.zeros((n, windows), dtype=torch.int64, device=rows.device)
    for k in range(KMER):
        code = code * 4 + (rows[:, k:k + windows].long() - 1).clamp(min=0)
    ok = torch.arange(windows, device=rows.device)[None, :] < (lens - KMER + 1)[:, None]
    counts = torch.zeros((n, 4 ** KMER), dtype=torch.int16, device=rows.device)
    return counts.scatter_add_(1, code, ok.to(torch.int16)), code, ok


def runs_of_three(rows):
    same = (rows[..., 1:] == rows[..., :-1]) & (rows[..., 1:] > 0)
    run = torch.zeros(rows.shape, dtype=torch.bool, device=rows.device)
    run3 = same[..., 1:] & same[..., :-1]
    for s in range(3):
        run[..., s:rows.shape[-1] - 2 + s] |= run3
    return run


def aligned_rows(center, rows, lens, band: int, homo_gap: int):
    """Ends-free banded alignment of the center with every row, all rows at
    once along the anti-diagonals; ties go up, left, diagonal. Gives for each
    row position the center's code there, 0 at an insertion."""
    dev, n = rows.device, rows.shape[0]
    l1 = center.numel()
    l2, tmax = lens, l1 + int(lens.max())
    lo, hi = -(band + (l1 - l2).clamp(min=0)), band + (l2 - l1).clamp(min=0)
    offs = torch.arange(int(lo.min()), int(hi.max()) + 1, device=dev)
    width = offs.numel()
    band_ok = (offs >= lo[:, None]) & (offs <= hi[:, None])
    gap1 = torch.where(runs_of_three(center), homo_gap, -8).int()
    gap2 = torch.where(runs_of_three(rows), homo_gap, -8).int()
    neg = torch.full((n, 1), -9999, dtype=torch.int32, device=dev)
    two = one = neg.expand(n, width)
    moves = torch.zeros((tmax + 1, n, width), dtype=torch.uint8, device=dev)
    for t in range(tmax + 1):
        i, j = torch.div(t - offs, 2, rounding_mode="floor"), torch.div(t + offs, 2, rounding_mode="floor")
        on = ((t - offs) % 2 == 0) & (i >= 0) & (i <= l1) & (j >= 0)
        ok = band_ok & on & (j <= l2[:, None])
        inner = ok & (i > 0) & (j > 0)
        ic, jc = (i - 1).clamp(0, l1 - 1), (j - 1).clamp(0, rows.shape[1] - 1)
        up = torch.cat([one[:, 1:], neg], 1) + torch.where(j == l2[:, None], 0, gap1[ic])
        left = torch.cat([neg, one[:, :-1]], 1) + torch.where(i == l1, 0, gap2[:, jc])
        diag = two + torch.where(center[ic] == rows[:, jc], 5, -4)
        best = torch.maximum(torch.maximum(up, left), diag)
        moves[t] = torch.where(up == best, 3, torch.where(left == best, 2, 1)).to(torch.uint8)
        two, one = one, torch.where(inner, best, torch.where(ok, 0, -9999)).int()
    out = torch.zeros(rows.shape, dtype=torch.int8, device=dev)
    i, j, at = torch.full((n,), l1, device=dev), l2.clone(), torch.arange(n, device=dev)
    for _ in range(tmax):
        v = moves[i + j, at, (j - i - offs[0]).clamp(0, width - 1)].long()
        v = torch.where(i == 0, 2, torch.where(j == 0, 3, v))
        done = (i == 0) & (j == 0)
        hit = (v == 1) & ~done
        out[at[hit], j[hit] - 1] = center[i[hit] - 1].to(torch.int8)
        i = torch.where(done | (v == 2), i, i - 1)
        j = torch.where(done | (v == 3), j, j - 1)
    return out


def exact_call(case: dict, rows, lens, count, mean, center: int, cutoff: float):
    """lambda of every unique against one center (0 where it is not compared)."""
    err, ncol = model_of(case)
    model = torch.from_numpy(err).to(rows.device)
    band, homo = (32, -1) if case.get("long") else (16, -8)
    counts, code, ok = kmer_counts(rows, lens)
    shared = torch.cat([torch.minimum(part, counts[center]).sum(1) for part in counts.split(50000)]).double()
    shorter = torch.minimum(lens, lens[center]).double() - KMER + 1
    kdist = 1.0 - shared / shorter
    use = (count <= count[center]) & ~(kdist > cutoff)
    same = lens == lens[center]
    equal = ((code == code[center]) & ok).sum(1).double()
    gapless = same & (torch.abs(1.0 - equal / shorter - kdist) < 2.220446049250313e-16)
    lam = torch.zeros(len(lens), dtype=torch.float64, device=rows.device)
    ref = rows[center, :int(lens[center])]
    for part in use.nonzero()[:, 0].split(1500 if case.get("long") else 20000):
        sub, n = rows[part], lens[part]
        by = torch.zeros_like(sub)
        by[:] = rows[center]
        dp = (~gapless[part]).nonzero()[:, 0]
        if len(dp):
            by[dp] = aligned_rows(ref, sub[dp], n[dp], band, homo)
        by = torch.where(by > 0, by, sub).long() - 1
        row = by.clamp(min=0) * 4 + (sub.long() - 1).clamp(min=0)
        p = model[row, mean[part].long().clamp(max=ncol - 1)]
        lam[part] = torch.where(sub > 0, p, 1.0).prod(1)
    return lam


def exact(case: dict, seed: int):
    """The lambdas of the compare calls; a denoising's tables follow from
    thousands of decisions and have no closed form here."""
    if case["kind"] not in ("map", "store"):
        return None
    rows, lens, count, mean = encoded(case, seed)
    other = late_center(rows, lens, count)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
           (rows.view(np.int8), lens.astype(np.int64), count.astype(np.int64), mean)]
    if case["kind"] == "map":
        lam = exact_call(case, *dev, *((other, CUTOFF) if case.get("late") else (0, 1.0)))
        return lam.cpu().numpy(), None, None, None
    total = float(dev[2].sum())
    e = torch.full((len(lens),), -999.0, dtype=torch.float64, device=dev[0].device)
    calls = []
    for center, cutoff in ((0, 1.0), (other, CUTOFF)):
        lam = exact_call(case, *dev, center, cutoff)
        kept = lam * total > e
        e = torch.where(kept, torch.maximum(e, lam * float(count[center])), e)
        calls.append({"index": None, "lambda": padded(lam[kept].cpu().numpy(), len(lens)), "hamming": None,
                      "self": float(lam[center]), "counters": None})
    return {"first": calls[0], "later": calls[1], "e_minmax": e.cpu().numpy()}
