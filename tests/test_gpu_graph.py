"""The batched form: a correction round captured as one CUDA graph and replayed
gives the same bytes as the plain form, and re-plans when the reads change."""
import pytest
from fixtures import FIXTURES, params, upper
from hero_testlib import assert_same_consensus

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["c1_20k", "c2_30k", "mix_i0"])
def test_graph_rounds_match_plain(gpu_lib, oracle, name):
    from hero_b200 import Hero
    gen, flags = FIXTURES[name]
    rs = upper(gen())
    kw = params(flags)
    want = oracle.correct(rs, **kw)
    with Hero(subject_batch=1500, **kw) as h:  # several batches inside one graph
        h.set_queries(rs.seq, rs.off, rs.names)
        for rnd in range(4):                      # eager+capture, then 3 replays
            h.round(graph=True)
            got = h.fetch()
            assert_same_consensus(want, got, f"{name} round {rnd}")
        assert h.stats()["graph_rounds"] == 3
        h.round(graph=False)                      # plain form on the same context
        assert_same_consensus(want, h.fetch(), f"{name} plain")


def test_graph_replans_when_reads_change(gpu_lib, oracle):
    from hero_b200 import Hero
    a = upper(FIXTURES["c1_20k"][0]())
    b = upper(FIXTURES["mix"][0]())
    with Hero() as h:
        for rs in (a, b, a):
            h.set_queries(rs.seq, rs.off, rs.names)
            h.round(graph=True)
            h.round(graph=True)
            assert_same_consensus(oracle.correct(rs), h.fetch(), "replan")


def test_replays_count_their_own_batches(gpu_lib, oracle):
    """Alignments between replays, in more batches than the captured round's, leave
    its statistics and its results as they were."""
    import numpy as np
    from hero_b200 import Hero
    rs = upper(FIXTURES["c1_20k"][0]())
    want = oracle.correct(rs)
    n = 60 * rs.n  # short subjects, so that no buffer has to grow
    pieces = np.concatenate([rs.seq[int(a):int(a) + 45] for a in rs.off[:rs.n]])
    assert len(pieces) == 45 * rs.n
    fields = ("subjects", "dp_segments", "chains_kept")
    with Hero(subject_batch=1500, **params([])) as h:
        h.set_queries(rs.seq, rs.off, rs.names)
        h.round(graph=True)
        first = h.stats()
        h.align_subjects(np.tile(pieces, 60), np.arange(n + 1, dtype=np.uint64) * np.uint64(45),
                         np.arange(1, n + 1, dtype=np.int64) + 10**6)
        for rnd in range(2):
            before = h.stats()
            h.round(graph=True)
            after = h.stats()
            assert_same_consensus(want, h.fetch(), f"round {rnd}")
            assert [after[f] - before[f] for f in fields] == [first[f] for f in fields]
        assert after["graph_rounds"] == 2
        assert after["ms_dp_kernel"] - before["ms_dp_kernel"] < 1000
