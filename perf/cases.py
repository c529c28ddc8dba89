"""The work a user has this framework do, as timed cases.

Every case is one call sequence through the package's public entry points
(hero_b200.Hero, hero_b200._lib.HeroServer) on seeded synthetic reads: a
correction of a read set against itself (HERO's -q X -s X -c), its rounds as a
replayed graph, the alignment output (no -c), --merge, --mapping with streamed
subject reads, and the served form.  Read lengths, coverages, error models and
flags are those of hero_b200.synth, the golden fixtures and bench.py; the
reads are generated here on the GPU because they are made many times.

Where a program that cares for throughput keeps page-locked buffers the case
does too (io "pinned": the raw-pointer calls bench.py's end-to-end number
uses); the small ones pass and receive plain arrays.
"""
import ctypes
import math

import numpy as np
import torch

from hero_b200._lib import Hero, HeroServer

ACGT = torch.tensor([65, 67, 71, 84], dtype=torch.uint8)  # A C G T; complement of code c is 3 - c
RESULT = (("seq", torch.uint8), ("imin", torch.int32), ("imed", torch.int32),
          ("imax", torch.int32), ("mismatch_rate", torch.float64), ("gc", torch.float64),
          ("good", torch.uint8))


def _case(name, mode, aligner, genome_bp, coverage, lmin, lmax, errors, **more):
    """One case.  errors: "sub" = 1 % iid substitutions (the plain method's reads),
    "ramp" = substitutions rising 0.1 % -> 2 % along the read and short indels (the
    affine workloads' reads).  mis / indel: -m / -i as rates (1.0 = HERO's default)."""
    c = dict(mode=mode, aligner=aligner, genome_bp=genome_bp, coverage=coverage, lmin=lmin,
             lmax=lmax, errors=errors, repeats=0, n_bases=0.0, k=39, min_overlap=40, mis=1.0,
             indel=1.0, threshold=0.6, io="pinned", chunks=1, jobs=1)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a handful of reads, a locus or an amplicon: launches and host calls are all there is
        _case("tiny_100", "correct", "global", 1000, 30.0, 100, 100, "sub", io="arrays"),
        # a small ragged job with a few N bases (uneven lengths, odd counts), affine
        _case("small_75_250", "correct", "affine", 20011, 35.0, 75, 250, "ramp", n_bases=0.01,
              io="arrays"),
        # the headline workload: 300 k x 100 bp at 30x, global aligner, host reads to host results
        _case("plain_100", "correct", "global", 1000000, 30.0, 100, 100, "sub"),
        # the affine/indel workload at full size: 5 Mbp with repeats, 1.67 M x 150 bp (the largest)
        _case("affine_150", "correct", "affine", 5000000, 50.0, 150, 150, "ramp", repeats=40),
        # uneven read lengths at high coverage, as the mixed-length workload
        _case("mixed_75_250", "correct", "affine", 400000, 100.0, 75, 250, "ramp"),
        # strict -m 3 -i 2 (the narrow-band fixtures' flags): bands of a few diagonals, early exits
        _case("narrow_150", "correct", "affine", 300000, 40.0, 150, 150, "ramp", mis=0.03,
              indel=0.02),
        # reads of 300-600 bp (merged pairs and longer chemistries; HERO's own limit is 700)
        _case("long_300_600", "correct", "affine", 100000, 30.0, 300, 600, "ramp"),
        # the headline workload device-resident, the batched form: one replayed graph a round
        _case("round_100", "round", "global", 1000000, 30.0, 100, 100, "sub"),
        # HERO without -c: the .aln text of every read's records
        _case("alignments_150", "alignments", "affine", 200000, 40.0, 150, 150, "ramp",
              io="arrays"),
        # --merge: read pairs of fragments of 160-290 bp, corrected and merged
        _case("merge_150", "merge", "affine", 1000000, 50.0, 150, 150, "sub"),
        # --mapping with k = 31: other reads streamed against the query set in three chunks
        _case("mapping_250", "mapping", "global", 300000, 20.0, 250, 250, "ramp", k=31, chunks=3,
              io="arrays"),
        # the served form: eight independent jobs of 100, 150 and 250 bp reads queued at once
        _case("served_8", "serve", "affine", 60000, 50.0, 100, 250, "ramp", jobs=8, io="arrays"),
    ]


MODES = ("correct", "correct", "correct", "correct", "round", "alignments", "merge", "mapping",
         "serve")


def draw(rng):
    """One more case: mode, aligner, flags, lengths and coverage over their ranges, the genome
    log-uniform from a locus to a few Mbp (bounded so that no draw costs more than the largest
    listed case)."""
    mode = rng.choice(MODES)
    aligner = rng.choice(("affine", "affine", "global"))
    shape = rng.random()
    if mode == "merge":
        lmin = lmax = rng.randint(100, 150)
    elif shape < 0.45:
        lmin = lmax = rng.choice((100, 150, 250, rng.randint(75, 260)))
    elif shape < 0.9:
        lmin = rng.randint(50, 120)
        lmax = rng.randint(lmin + 20, 260)
    else:
        lmin = rng.randint(200, 300)
        lmax = rng.randint(350, 600)
    c = _case(None, mode, aligner, 0, round(rng.uniform(20, 80), 2), lmin, lmax,
              "sub" if aligner == "global" and rng.random() < 0.7 else "ramp",
              k=rng.choice((39, 39, 39, 31, 21)), threshold=rng.choice((0.6, 0.6, 0.7)),
              min_overlap=rng.choice((40, 40, 60)),
              n_bases=rng.choice((0.0, 0.0, 0.01)) if mode != "merge" else 0.0,
              io=rng.choice(("arrays", "pinned")) if mode in ("correct", "merge") else
              ("pinned" if mode == "round" else "arrays"),
              chunks=rng.randint(1, 4) if mode == "mapping" else 1,
              jobs=rng.randint(2, 9) if mode == "serve" else 1)
    if rng.random() < 0.2:
        c["mis"], c["indel"] = rng.choice((0.02, 0.03, 0.04)), rng.choice((0.0, 0.01, 0.02))
    c["genome_bp"] = 1
    # the cell estimate is proportional to the genome: at most 20 G cells a draw (the largest
    # listed case has more than ten times that), 2 G for long reads and served jobs
    most = (2e9 if lmax > 260 or mode == "serve" else 2e10) / max(1.0, _cells(c))
    hi = min(3e6, max(2000.0, most))
    c["genome_bp"] = int(math.exp(rng.uniform(math.log(2 * lmax + 1000), math.log(hi + 2 * lmax + 1000))))
    if mode in ("correct", "round") and c["genome_bp"] > 200000 and rng.random() < 0.3:
        c["repeats"] = rng.randint(4, 40)
    return c


# ---------------------------------------------------------------------------
# reads
# ---------------------------------------------------------------------------
def _genome(g, bp, repeats):
    a = torch.randint(0, 4, (bp,), generator=g, device="cuda", dtype=torch.uint8)
    if repeats:  # diverged copies of segments, as the affine workload's genome
        lmax = min(5000, max(1000, bp // 20))
        u = torch.rand((repeats, 3), generator=g, device="cuda").tolist()
        for x, y, z in u:
            ln = int(1000 + x * (lmax - 1000))
            src, dst = int(y * (bp - ln)), int(z * (bp - ln))
            seg = a[src:src + ln].clone()
            hit = torch.rand(ln, generator=g, device="cuda") < 0.005
            step = torch.randint(1, 4, (ln,), generator=g, device="cuda", dtype=torch.uint8)
            a[dst:dst + ln] = torch.where(hit, (seg + step) & 3, seg)
    return a


def _substitute(g, code, rate):
    hit = torch.rand(code.shape, generator=g, device="cuda") < rate
    step = torch.randint(1, 4, code.shape, generator=g, device="cuda", dtype=torch.uint8)
    return torch.where(hit, (code + step) & 3, code)


def _sample(g, genome, n, lmin, lmax, errors, n_bases):
    """n reads from random places and strands: flat ASCII (on the device) and lengths."""
    # the lengths are the case's own: every seed's read set has the same size
    own = torch.Generator(device="cuda")
    own.manual_seed(n)
    lens = torch.randint(lmin, lmax + 1, (n,), generator=own, device="cuda")
    slack = 48
    acgt = ACGT.cuda()
    flat = []
    for a in range(0, n, 100_000):
        ln = lens[a:a + 100_000]
        m = len(ln)
        col = torch.arange(lmax, device="cuda")
        start = torch.randint(0, max(1, len(genome) - lmax - slack), (m,), generator=g, device="cuda")
        rc = torch.rand(m, generator=g, device="cuda") < 0.5
        adv = torch.ones((m, lmax), dtype=torch.int32, device="cuda")
        inserted = torch.zeros((m, lmax), dtype=torch.bool, device="cuda")
        if errors == "ramp":  # indels: 0.05 % of each a base, 1-3 bases long
            ev = torch.rand((m, lmax), generator=g, device="cuda")
            size = 1 + torch.randint(0, 2, (m, lmax), generator=g, device="cuda", dtype=torch.int32) \
                * torch.randint(0, 3, (m, lmax), generator=g, device="cuda", dtype=torch.int32)
            adv += torch.where(ev < 0.0005, size, 0)
            ins = torch.where((ev >= 0.0005) & (ev < 0.001), size, 0)
            for d in range(3):
                inserted[:, d:] |= ins[:, :lmax - d] > d
            adv = torch.where(inserted, 0, adv)
        src = torch.clamp(torch.cumsum(adv, 1) - 1, 0, lmax + slack - 1)
        src = torch.where(rc[:, None], start[:, None] + (lmax + slack - 1) - src, start[:, None] + src)
        src = torch.clamp(src, max=len(genome) - 1)
        code = genome[src]
        code = torch.where(rc[:, None], 3 - code, code)
        if errors == "ramp":
            code = torch.where(inserted, torch.randint(0, 4, code.shape, generator=g, device="cuda",
                                                       dtype=torch.uint8), code)
            rate = 0.001 + 0.019 * col[None, :] / (ln[:, None] - 1)
        else:
            rate = torch.full((1, 1), 0.01, device="cuda")
        base = acgt[_substitute(g, code, rate).long()]
        if n_bases:  # an N in this fraction of the reads
            has = torch.rand(m, generator=g, device="cuda") < n_bases
            at = (torch.rand(m, generator=g, device="cuda") * ln).long()
            rows = torch.nonzero(has)[:, 0]
            base[rows, at[rows]] = ord("N")
        flat.append(base[col[None, :] < ln[:, None]])
    return torch.cat(flat), lens


def _pairs(g, genome, n, length):
    """Read pairs of fragments of 160-290 bases (at least a read long), 0.5 % substitutions."""
    np_ = max(1, n // 2)
    flen = torch.randint(max(160, length), 291, (np_,), generator=g, device="cuda")
    start = (torch.rand(np_, generator=g, device="cuda", dtype=torch.float64) * (len(genome) - flen)).long()
    col = torch.arange(length, device="cuda")
    head = genome[start[:, None] + col]
    tail = 3 - genome[(start + flen)[:, None] - 1 - col]
    flip = torch.rand(np_, generator=g, device="cuda") < 0.5
    both = torch.stack([torch.where(flip[:, None], tail, head),
                        torch.where(flip[:, None], head, tail)], 1).reshape(2 * np_, length)
    lens = torch.full((2 * np_,), length, device="cuda")
    return ACGT.cuda()[_substitute(g, both, 0.005).long()].reshape(-1), lens


def _count(case, genome_bp=None):
    mean = (case["lmin"] + case["lmax"]) / 2
    n = max(2, round(case["coverage"] * (genome_bp or case["genome_bp"]) / mean))
    return n + (n & 1) if case["mode"] == "merge" else n


def _host(seq, lens, pinned, first=1):
    """A read set in host memory: bases, offsets, ids (numpy views)."""
    n = len(lens)
    off = torch.zeros(n + 1, dtype=torch.int64)
    off[1:] = torch.cumsum(lens, 0).cpu()
    uid = torch.arange(first, first + n, dtype=torch.int64)
    out = []
    for t in (seq, off, uid):
        h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned)
        h.copy_(t)
        out.append(h.numpy())
    return out[0], out[1].view(np.uint64), out[2]


def _read_sets(case, seed):
    """The case's read sets in host memory: one, one a job, or queries and subject chunks."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    pinned = case["io"] == "pinned"
    shape = (case["lmin"], case["lmax"], case["errors"], case["n_bases"])
    if case["mode"] == "serve":
        sets = []
        for j in range(case["jobs"]):  # sizes around the mean, one read length a job
            bp = int(case["genome_bp"] * (0.3 + 1.4 * j / max(1, case["jobs"] - 1)))
            length = max(case["lmin"], (100, 150, 250)[j % 3]) if case["lmax"] >= 250 else case["lmin"]
            bp = max(bp, 4 * length + 200)
            genome = _genome(g, bp, 0)
            n = max(2, int(case["coverage"] * bp / length))
            sets.append(_host(*_sample(g, genome, n, length, length, *shape[2:]), pinned))
        return sets
    genome = _genome(g, max(case["genome_bp"], 2 * case["lmax"] + 200), case["repeats"])
    n = _count(case)
    if case["mode"] == "merge":
        return [_host(*_pairs(g, genome, n, case["lmax"]), pinned)]
    sets = [_host(*_sample(g, genome, n, *shape), pinned)]
    if case["mode"] == "mapping":
        per = n // case["chunks"] + 1
        for j in range(case["chunks"]):
            sets.append(_host(*_sample(g, genome, per, *shape), pinned, n + 1 + j * per))
    return sets


class State:
    """Reads in host memory, and the handle (and page-locked result buffers) a program keeps."""

    def __init__(self, case, seed):
        self.mode, self.io = case["mode"], case["io"]
        self.sets = _read_sets(case, seed)
        args = dict(k=case["k"], min_overlap=case["min_overlap"], aligner=case["aligner"],
                    max_mismatch_rate=case["mis"], max_indel_rate=case["indel"],
                    consensus_threshold=case["threshold"])
        if self.mode == "serve":
            self.handle = HeroServer(**args)
            return
        self.handle = Hero(alignment_output=self.mode == "alignments",
                           merge_pairs=self.mode == "merge", mapping=self.mode == "mapping", **args)
        seq, off, _ = self.sets[0]
        if self.io == "pinned":
            self.out = {f: torch.empty(len(seq) if f == "seq" else len(off) - 1, dtype=t,
                                       pin_memory=True) for f, t in RESULT}
            self.where = [self.out[f].data_ptr() for f, _ in RESULT]
        if self.mode == "alignments":  # room for the text: 50 characters a record, and spare
            self.text = np.zeros(4096 + int(150 * _records(case)), np.uint8)
        if self.mode == "round":
            self.handle.set_queries(*self.sets[0])

    def __del__(self):
        if getattr(self, "handle", None):
            self.handle.close()


def prepare(case, seed):
    return State(case, seed)


def _load(s):
    seq, off, uid = s.sets[0]
    if s.io == "pinned":
        s.handle.set_queries_ptr(seq.ctypes.data, off.ctypes.data, uid.ctypes.data, len(off) - 1,
                                 len(seq))
    else:
        s.handle.set_queries(seq, off, uid)
    s.handle.build_index()


def run(s):
    h = s.handle
    if s.mode == "serve":
        ids = [h.submit(*r) for r in s.sets]
        got = []
        for j in ids:
            h.wait(j)
            got.append(h.result(j))
            h.release(j)
        return got
    if s.mode == "round":
        h.round(graph=True)
        h.fetch_ptr(*s.where)
        return s.out
    _load(s)
    if s.mode == "mapping":
        for chunk in s.sets[1:]:
            h.align_subjects(*chunk)
        hist = np.zeros(4096, np.uint64)  # of the same size for every read set
        got = h.mapping_histogram()
        hist[:len(got)] = got
        return {"histogram": hist}
    h.align_self()
    if s.mode == "alignments":  # the C ABI's calls: the text goes straight to the program's buffer
        n = ctypes.c_uint64()
        if h.lib.hero_alignments_size(h.h, ctypes.byref(n)) or \
                h.lib.hero_alignments_take(h.h, s.text.ctypes.data, len(s.text)):
            raise RuntimeError("alignments: %d bytes of text" % n.value)
        return {"aln": s.text, "bytes": n.value}
    if s.io == "pinned":
        h.consensus_ptr(*s.where)
        res = dict(s.out)
    else:
        res = h.consensus()
    if s.mode == "merge":
        res.update(h.merge_pairs())
    return res


def _records(case, L=None):
    """Alignment records of a pass, estimated: both sides of every overlap of a k-mer or more."""
    L = L or (case["lmin"] + case["lmax"]) / 2
    reads = case["coverage"] * case["genome_bp"] / L * case["jobs"]
    return reads * 2 * case["coverage"] * max(1.0, L - case["k"]) / L


def _cells(case):
    """Cells of the banded DP of a pass, estimated: those of a record from the read length
    (0.22 (L - k)^2 on the repository's workloads; fewer where -i narrows the band)."""
    ls = [(case["lmin"] + case["lmax"]) / 2]
    if case["mode"] == "serve" and case["lmax"] >= 250:
        ls = [100, 150, 250]
    total = 0.0
    for L in ls:
        side = max(1.0, L - case["k"])
        cells = 0.22 * side * side
        if case["indel"] < 0.5:
            m = 2 * round(0.7 * L * case["indel"])
            cells = min(cells, 0.5 * side * (2 * m + 1))
        total += _records(case, L) * cells
    return total / len(ls)


def work(case):
    """Reads in (bases, offsets, ids), results out, and the DP's integer operations (10 a cell for
    the affine recurrence, 6 for the global one)."""
    bases = case["coverage"] * case["genome_bp"] * case["jobs"]
    reads = bases / ((case["lmin"] + case["lmax"]) / 2)
    moved = bases + 16 * reads
    if case["mode"] == "alignments":  # about ten characters of text a base
        moved += 10 * bases
    elif case["mode"] == "mapping":
        moved *= 2
    else:
        moved += bases * (2 if case["mode"] == "merge" else 1) + 29 * reads
    return {"bytes": moved, "flops": _cells(case) * (10 if case["aligner"] == "affine" else 6)}


def exact(case, seed):
    """The GC content of each read is the one result that plain 64-bit arithmetic gives (a count
    over a length); every other output is whole numbers, or a quotient of whole numbers that only
    the alignments give."""
    if case["mode"] in ("alignments", "mapping"):
        return None
    got = []
    for seq, off, _ in _read_sets(case, seed):
        at = off.astype(np.int64)
        n = np.concatenate([[0], np.cumsum((seq == ord("G")) | (seq == ord("C")))])
        d = {f: None for f, _ in RESULT}
        d["gc"] = (n[at[1:]] - n[at[:-1]]) / (at[1:] - at[:-1])
        if case["mode"] == "merge":
            d.update(merged_seq=None, merged_len=None)
        got.append(d)
    return got if case["mode"] == "serve" else got[0]
