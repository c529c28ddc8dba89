"""The window DP (hero_band.cuh): whatever its certificate accepts is the
whole-matrix path, move for move.

On the CPU the header's item logic runs beside hero_core.cuh's whole-matrix DP
on every pair of short strings and on random segments of the kinds that strain
the certificate (tandem repeats, two-letter strings, indels, narrow bands); on
the GPU the kernels run on segments at the edges of their classes against the
oracle."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
from hero_testlib import ROOT

SRC = os.path.join(ROOT, "tests", "emu", "band_emu.cpp")
LIB = os.path.join(ROOT, "_build", "libband_emu.so")
HDRS = [os.path.join(ROOT, "hero_b200", "csrc", h) for h in ("hero_band.cuh", "hero_core.cuh")]
ACGT = np.frombuffer(b"ACGT", np.uint8)


@pytest.fixture(scope="module")
def band():
    if not os.path.exists(LIB) or any(os.path.getmtime(s) > os.path.getmtime(LIB) for s in [SRC] + HDRS):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-o", LIB, SRC], check=True)
    return C.CDLL(LIB)


def _clean(counts):
    segments, certified, straight, ops, sums, straight_ops = counts
    assert (ops, sums, straight_ops) == (0, 0, 0), counts
    return segments, certified, straight


# nb 0: the segments finished without a window (at most one mismatch on the main diagonal);
# nb < 0: the wide window of -nb diagonals
@pytest.mark.parametrize("affine,nb", [(1, 0), (1, 4), (1, 8), (1, 16), (1, -10), (0, 0), (0, 4), (0, 8), (0, -10)])
@pytest.mark.parametrize("kind", [0, 1, 2], ids=["both", "right", "left"])
def test_every_short_segment(band, affine, nb, kind):
    n = np.zeros(3, np.int64)
    for letters, total in ((2, 11), (3, 7), (4, 6)):
        for rows in range(1, total):
            for cols in range(1, min(rows, total - rows) + 1):
                for mask, m in ((0, 65535), (1, 0), (1, 1), (1, 3)):
                    c = (C.c_uint64 * 6)()
                    band.band_exhaustive(affine, nb, kind, mask, letters, rows, cols, C.c_int64(m), c)
                    n += _clean(list(c))
    assert n[1] > n[2] and n[1] > n[0] // (4 if nb else 50)  # it accepts, and not only the plainest paths


@pytest.mark.parametrize("affine,nb", [(1, 0), (1, 11), (1, 16), (1, 19), (1, 24), (1, 26), (1, 40), (1, -10), (1, -64),
                                       (1, -136), (0, 0), (0, 8), (0, 16), (0, -10), (0, -64), (0, -136)])
@pytest.mark.parametrize("cmax", [5, 40, 250, 1023])
def test_random_segments(band, affine, nb, cmax):
    for mask, m in ((0, 0), (1, 4), (1, 30)) if nb >= 0 else ((0, 0),):  # the wide window takes whole bands
        c = (C.c_uint64 * 6)()
        band.band_random(affine, nb, mask, C.c_uint64(nb * 1000 + cmax), C.c_uint64(200000 // (cmax + 100)), cmax,
                         C.c_int64(m), c)
        segments, certified, straight = _clean(list(c))
        assert segments and certified > straight


def test_dp_pieces_of_a_chain_counted_without_walking_it(band):
    band.chain_counts.restype = C.c_uint64
    assert band.chain_counts(C.c_uint64(3), C.c_uint64(200000)) == 0


def test_keys_of_packed_windows(band):
    band.window_keys.restype = C.c_uint64
    assert band.window_keys(C.c_uint64(5)) == 0


def _segments(rng, n):
    """(subject, query, band, flags): copies with e substitutions and at times an
    indel, on either side, with a free run on the anchored side's far end."""
    out = []
    sizes = [1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 64, 111, 211, 255, 256, 257]
    for i in range(n):
        c = int(sizes[i % len(sizes)])
        e = i // len(sizes) % 7
        kind = int(rng.integers(0, 3))
        col = ACGT[rng.integers(0, 4, c)]
        row = col.copy()
        for p in rng.integers(0, c, e):
            row[p] = ACGT[rng.integers(0, 4)]
        if rng.random() < 0.3:
            p, k = int(rng.integers(0, c)), int(rng.integers(1, 4))
            row = np.concatenate([row[:p], ACGT[rng.integers(0, 4, k)], row[p:]]) if rng.random() < 0.5 or c < 8 \
                else np.delete(row, slice(p, p + k))
        d = int(rng.integers(0, 70)) if kind else 0
        free = ACGT[rng.integers(0, 4, d)] if rng.random() < 0.7 else np.resize(col, d)
        row = np.concatenate([free, row] if kind == 1 else [row, free])
        s, q = (row, col) if rng.random() < 0.5 else (col, row)
        out.append((bytes(s), bytes(q), int(rng.choice([2, 5, 9, 300])), kind))
    return out


def _long_segments(rng, n):
    """Segments of up to 800 rows and 600 columns: copies with many mismatches and
    gaps (the wide window), and unrelated strings (whole matrices, in panels)."""
    out = []
    for i in range(n):
        c = int(rng.choice([100, 129, 255, 256, 257, 263, 264, 511, 512, 513, 600]))
        kind = int(rng.integers(0, 3))
        col = ACGT[rng.integers(0, 4, c)]
        row = col.copy() if i % 4 else ACGT[rng.integers(0, 4, c)]
        for p in rng.integers(0, c, int(rng.integers(0, 25))):
            row[p] = ACGT[rng.integers(0, 4)]
        for _ in range(int(rng.integers(0, 5))):
            p, k = int(rng.integers(0, len(row))), int(rng.integers(1, 12))
            row = np.concatenate([row[:p], ACGT[rng.integers(0, 4, k)], row[p:]]) if rng.random() < 0.5 \
                else np.delete(row, slice(p, p + k))
        d = int(rng.integers(0, 200)) if kind else 0
        free = ACGT[rng.integers(0, 4, d)]
        row = np.concatenate([free, row] if kind == 1 else [row, free])
        s, q = (row, col) if rng.random() < 0.5 else (col, row)
        out.append((bytes(s), bytes(q), int(rng.choice([20, 900, 900])), kind))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("affine", [0, 1])
@pytest.mark.parametrize("make,count", [(_segments, 5000), (_long_segments, 300), (_long_segments, 7)])
def test_gpu_segments_at_the_edges_of_the_classes(gpu_lib, oracle, affine, make, count):
    from hero_b200 import Hero
    seg = make(np.random.default_rng(40 + affine), count)
    n = len(seg)
    off = [np.zeros(n + 1, np.uint64) for _ in range(2)]
    for h in range(2):
        off[h][1:] = np.cumsum([len(x[h]) for x in seg])
    seq = [np.frombuffer(b"".join(x[h] for x in seg), np.uint8) for h in range(2)]
    idx, zeros = np.arange(n, dtype=np.uint32), np.zeros(n, np.int32)
    with Hero() as h:
        ops, oo, nops = h.align_segments(affine, seq[0], off[0], seq[1], off[1], idx, np.zeros(n, np.uint8), idx,
                                         zeros, np.diff(off[0]).astype(np.int32), zeros,
                                         np.diff(off[1]).astype(np.int32), np.array([x[3] for x in seg], np.uint8),
                                         np.array([x[2] for x in seg], np.int64))
    for i, (s, q, m, kind) in enumerate(seg):
        want, _ = oracle.align(affine, s, q, m, kind == 1, kind == 2)
        got = ops[int(oo[i]):int(oo[i]) + int(nops[i])]
        assert np.array_equal(got, want), (i, len(s), len(q), m, kind)


def _correct(h, rs):
    h.set_queries(rs.seq, rs.off, rs.names)
    h.build_index()
    h.align_self()
    return h.consensus()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["c1_20k", "c2_30k"])
def test_gpu_budgets_without_room_for_the_windows(gpu_lib, oracle, name):
    """Whatever buffer meets the budget first, the windows' memory goes and the
    result stays, or the job is refused."""
    from fixtures import FIXTURES, params, upper
    from hero_b200 import Hero, HeroError
    from hero_testlib import assert_same_consensus
    gen, flags = FIXTURES[name]
    rs, kw = upper(gen()), params(flags)
    want = oracle.correct(rs, **kw)
    with Hero(subject_batch=500, **kw) as h:
        _correct(h, rs)
        peak, pairs = h.stats()["device_bytes_peak"], h.stats()["dp_cells_pairs"]
    done = without = 0
    for f in np.linspace(0.30, 1.0, 36):
        with Hero(subject_batch=500, device_memory_budget=int(peak * f), **kw) as h:
            try:
                got = _correct(h, rs)
            except HeroError as e:
                assert "OOM" in str(e)
                continue
            assert_same_consensus(want, got, f"{f:.2f} of the peak")
            done += 1
            without += h.stats()["dp_cells_pairs"] > pairs
    assert done and without


@pytest.mark.gpu
@pytest.mark.parametrize("plain", [False, True])
def test_gpu_graph_rounds_after_buffers_moved(gpu_lib, oracle, plain):
    """A captured round is captured again once a larger job has moved its buffers."""
    from fixtures import FIXTURES, upper
    from hero_b200 import Hero
    from hero_testlib import assert_same_consensus
    a, b = upper(FIXTURES["c1_20k"][0]()), upper(FIXTURES["mix"][0]())
    want = oracle.correct(a)
    with Hero() as h:
        h.set_queries(a.seq, a.off, a.names)
        h.round(graph=True)
        h.round(graph=True)
        off = np.concatenate([np.zeros(1, np.uint64)] + [b.off[1:] + np.uint64(i) * b.off[-1] for i in range(3)])
        h.align_subjects(np.tile(b.seq, 3), off, np.tile(b.names, 3))
        if plain:
            h.round(graph=False)
            assert_same_consensus(want, h.fetch(), "plain")
        for i in range(3):
            h.round(graph=True)
            assert_same_consensus(want, h.fetch(), f"round {i}")
        assert h.stats()["graph_rounds"] >= 3


def test_bases_are_read_inside_the_packed_arrays(tmp_path):
    """Segments at the ends of their read arrays, with free runs longer than the
    arrays' room, under address checking."""
    exe = str(tmp_path / "band_bounds")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address", "-o", exe,
                    os.path.join(ROOT, "tests", "emu", "band_bounds.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr[:3000]
    segments, certified, straight = map(int, r.stdout.split()[:3])
    assert certified > segments // 2 and straight > 1000


# the 16-bit halves of cells outside the aligner's band: a path 3000 points worse
# than all matches must not be certified, however much lies inside the window
@pytest.mark.parametrize("affine,nb", [(1, 16), (1, 24), (0, 16)])
@pytest.mark.parametrize("columns", [580, 620, 800, 900, 1023])
def test_cut_bands_beside_a_matching_diagonal(band, affine, nb, columns):
    n = np.zeros(3, np.int64)
    for m in (0, 1, 2):
        for shift in (m + 1, m + 2, m + 3):
            for period in (0, 2, 3, 4):
                for free in (0, 1):
                    c = (C.c_uint64 * 6)()
                    band.band_shifted(affine, nb, C.c_uint64(columns + 7 * shift + period), C.c_uint64(6), columns,
                                      C.c_int64(m), shift, period, free, c)
                    n += _clean(list(c))
    assert n[0]


def _check_segments(oracle, affine, seg, **kw):
    """hero_align_segments on (subject, query, band, flags) tuples against the oracle; returns the stats."""
    from hero_b200 import Hero
    n = len(seg)
    off = [np.zeros(n + 1, np.uint64) for _ in range(2)]
    for h in range(2):
        off[h][1:] = np.cumsum([len(x[h]) for x in seg])
    seq = [np.frombuffer(b"".join(x[h] for x in seg), np.uint8) for h in range(2)]
    idx, zeros = np.arange(n, dtype=np.uint32), np.zeros(n, np.int32)
    with Hero(**kw) as h:
        ops, oo, nops = h.align_segments(affine, seq[0], off[0], seq[1], off[1], idx, np.zeros(n, np.uint8), idx,
                                         zeros, np.diff(off[0]).astype(np.int32), zeros,
                                         np.diff(off[1]).astype(np.int32), np.array([x[3] for x in seg], np.uint8),
                                         np.array([x[2] for x in seg], np.int64))
        stats = h.stats()
    for i, (s, q, m, kind) in enumerate(seg):
        want, _ = oracle.align(affine, s, q, m, kind == 1, kind == 2)
        got = ops[int(oo[i]):int(oo[i]) + int(nops[i])]
        assert np.array_equal(got, want), (i, len(s), len(q), m, kind)
    return stats


@pytest.mark.gpu
@pytest.mark.parametrize("affine", [0, 1])
def test_gpu_cut_bands_beside_a_matching_diagonal(gpu_lib, oracle, affine):
    rng = np.random.default_rng(70 + affine)
    seg = []
    for c in (580, 620, 800, 900, 1023, 1024):
        for m in (0, 1, 2):
            for shift in (m + 1, m + 2, m + 3):
                for period in (0, 2, 3, 4):
                    kind = len(seg) % 3
                    col = ACGT[rng.integers(0, 4, c)] if not period else np.resize(ACGT[rng.integers(0, 4, period)], c)
                    new = ACGT[rng.integers(0, 4, shift)]
                    row = np.concatenate([new, col[:-shift]]) if len(seg) % 2 else np.concatenate([col[shift:], new])
                    free = ACGT[rng.integers(0, 4, len(seg) % 2 if kind else 0)]
                    row = np.concatenate([free, row] if kind == 1 else [row, free])
                    s, q = (row, col) if len(seg) % 5 else (col, row)
                    seg.append((bytes(s), bytes(q), m, kind))
    _check_segments(oracle, affine, seg)


def _moved_reads():
    """Pairs of 1000 bp reads: one the other with a base gone after 100, and behind
    it a substitution every 25 bases, so that they share no key there."""
    from hero_b200 import synth
    rng = np.random.default_rng(77)
    reads = []
    for _ in range(6):
        a = ACGT[rng.integers(0, 4, 1000)]
        b = np.concatenate([a[:100], a[101:], ACGT[rng.integers(0, 4, 1)]])
        for p in range(120, 1000, 25):
            b[p] = ACGT[(int(np.searchsorted(ACGT, b[p])) + 1) % 4]
        reads += [a, b, a, a]
    off = np.zeros(len(reads) + 1, np.uint64)
    off[1:] = np.cumsum([len(r) for r in reads])
    return synth.ReadSet(np.concatenate(reads), off, np.arange(1, len(reads) + 1, dtype=np.int64))


@pytest.mark.gpu
@pytest.mark.parametrize("aligner", ["affine", "global"])
def test_gpu_correction_with_no_indels_of_long_reads(gpu_lib, oracle, aligner):
    from hero_b200 import Hero
    from hero_testlib import assert_same_consensus
    rs, kw = _moved_reads(), dict(aligner=aligner, max_indel_rate=0.0)
    want = oracle.correct(rs, keep_segments=True, **kw)
    g = want["segments"]
    side = np.minimum(g["s1"] - g["s0"], g["q1"] - g["q0"])
    assert ((side > 800) & (side < 1000)).any()
    with Hero(**kw) as h:
        assert_same_consensus(want, _correct(h, rs), aligner)
        assert np.array_equal(h.votes(), want["votes"])


def _small_job():
    """700 reads of 250 bases, 56 k segments of up to 211 columns."""
    from hero_b200 import synth
    return synth.Job(0, 0.0, 5, 5000, 250, 35.0).reads()


@pytest.mark.gpu
def test_gpu_small_jobs_take_little_window_memory(gpu_lib):
    """The windows' codes follow the work: 400 warps of 135 KB and a quarter more
    here, 68 MB beside about 45 of other buffers (a warp for every 32 segments:
    272 MB)."""
    from hero_b200 import Hero
    rs = _small_job()
    with Hero(aligner="affine") as h:
        _correct(h, rs)
        st = h.stats()
    assert 20000 < st["dp_segments"] < 100000
    assert st["device_bytes_peak"] < 160e6


def _edited_segments(rng, n, columns):
    """Segments of the given numbers of columns: copies with many mismatches and gaps,
    every fourth an unrelated string."""
    out = []
    for i in range(n):
        c, kind = int(rng.choice(columns)), i % 3
        col = ACGT[rng.integers(0, 4, c)]
        row = col.copy() if i % 4 else ACGT[rng.integers(0, 4, c)]
        for p in rng.integers(0, c, int(rng.integers(4, 20))):
            row[p] = ACGT[rng.integers(0, 4)]
        for _ in range(int(rng.integers(1, 5))):
            p, k = int(rng.integers(0, len(row))), int(rng.integers(1, 12))
            row = np.concatenate([row[:p], ACGT[rng.integers(0, 4, k)], row[p:]])
        if len(row) < c + 1 or not kind:
            row = np.resize(row, c)
        free = ACGT[rng.integers(0, 4, int(rng.integers(0, 30)) if kind else 0)]
        row = np.concatenate([free, row] if kind == 1 else [row, free])
        s, q = (row, col) if rng.random() < 0.5 else (col, row)
        out.append((bytes(s), bytes(q), int(rng.choice([1500, 1500, 30])), kind))
    return out


# both widths of the wide window (8 lanes: the global aligner up to 256 columns, the
# affine one up to 64), and the hand-over to whole matrices past 1023 columns
@pytest.mark.gpu
@pytest.mark.parametrize("affine", [0, 1])
@pytest.mark.parametrize("columns,count", [([1, 8, 9, 63, 64], 1000), ([64, 65], 300), ([127, 128, 255, 256], 300),
                                           ([255, 256, 257], 200), ([1022, 1023, 1024, 1025], 120)])
def test_gpu_wide_windows_at_their_edges(gpu_lib, oracle, affine, columns, count):
    _check_segments(oracle, affine, _edited_segments(np.random.default_rng(80 + affine), count, columns))


@pytest.mark.gpu
@pytest.mark.parametrize("n,columns,free,budget", [(10, 50, 5, 13660160), (1000, 100, 20, 14622720), (20000, 100, 20, 35131392)])
def test_gpu_segments_without_room_for_the_windows(gpu_lib, n, columns, free, budget):
    """Segments take no more memory than whole matrices alone need (the budgets): what
    the windows have is given back, and the ops are the same."""
    from hero_b200 import Hero
    rng = np.random.default_rng(3)
    col = ACGT[rng.integers(0, 4, (n, columns))]
    row = np.concatenate([ACGT[rng.integers(0, 4, (n, free))], col], 1)
    col[:, ::9] = ACGT[rng.integers(0, 4, col[:, ::9].shape)]
    seq = [np.ascontiguousarray(x).reshape(-1) for x in (row, col)]
    off = [np.arange(n + 1, dtype=np.uint64) * np.uint64(x.shape[1]) for x in (row, col)]
    idx, zeros = np.arange(n, dtype=np.uint32), np.zeros(n, np.int32)
    got = []
    for limit in (0, budget):
        with Hero(device_memory_budget=limit) as h:
            ops, oo, nops = h.align_segments(1, seq[0], off[0], seq[1], off[1], idx, np.zeros(n, np.uint8), idx, zeros,
                                             np.diff(off[0]).astype(np.int32), zeros, np.diff(off[1]).astype(np.int32),
                                             np.ones(n, np.uint8), np.full(n, 1000, np.int64))
            got.append([bytes(ops[int(oo[i]):int(oo[i]) + int(nops[i])]) for i in range(n)])
    assert got[0] == got[1]
