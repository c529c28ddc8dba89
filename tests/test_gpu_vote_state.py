"""The vote state that contexts exchange: mismatch votes [bases][4], then the
match runs' differences, whose runs end at mismatches -- the same words from a
context's own memory and from the caller's."""
import numpy as np
import pytest
from fixtures import FIXTURES, params, upper
from hero_testlib import assert_same_consensus

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["c1_20k", "c2_30k", "mix_affine"])
def test_exchanged_words_are_the_votes(gpu_lib, oracle, name):
    import torch
    from hero_b200 import Hero
    gen, flags = FIXTURES[name]
    rs, kw = upper(gen()), params(flags)
    want = oracle.correct(rs, **kw)
    nb = int(rs.off[-1])
    own_words = torch.empty(5 * nb, dtype=torch.int32, device="cuda")
    ext = torch.zeros(5 * nb + 64, dtype=torch.int32, device="cuda")
    for buf in (None, ext):
        with Hero(**kw) as h:
            if buf is not None:
                h.set_vote_buffer(buf.data_ptr(), buf.numel() * 4)
            h.set_queries(rs.seq, rs.off, rs.names)
            h.build_index()
            h.align_self()
            if buf is None:
                h.votes_save(own_words.data_ptr())
            assert np.array_equal(h.votes(), want["votes"])
            assert_same_consensus(want, h.consensus(), name)
    words = own_words.cpu().numpy()
    assert np.array_equal(words, ext.cpu().numpy()[:5 * nb])
    votes, code = words[:4 * nb].view(np.uint32).reshape(nb, 4).copy(), np.full(256, 4)
    code[np.frombuffer(b"ACTG", np.uint8)] = np.arange(4)
    for a, b in zip(rs.off[:-1].astype(int), rs.off[1:].astype(int)):
        own = code[rs.seq[a:b]]
        runs = np.cumsum(words[4 * nb + a:4 * nb + b]).astype(np.uint32)
        ok = own < 4
        votes[np.arange(a, b)[ok], own[ok]] += runs[ok]
        assert not runs[~ok].any()
    assert np.array_equal(votes.reshape(-1), np.asarray(want["votes"], np.uint32).reshape(-1))


def test_captured_rounds_follow_the_vote_memory(gpu_lib, oracle):
    """A round captured with the context's own votes is captured again when the
    caller's memory takes their place, and the other way round, also with the
    same reads."""
    import torch
    from hero_b200 import Hero
    gen, flags = FIXTURES["c1_20k"]
    rs, kw = upper(gen()), params(flags)
    want = oracle.correct(rs, **kw)
    nb = int(rs.off[-1])
    ext = [torch.full((5 * nb,), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
    with Hero(**kw) as h:
        for buf in (None, ext[0], ext[1], None, ext[0]):
            before = [e.clone() for e in ext]
            h.set_vote_buffer(buf.data_ptr() if buf is not None else 0, 20 * nb if buf is not None else 0)
            h.set_queries(rs.seq, rs.off, rs.names)
            for rnd in range(3):
                h.round(graph=True)
                assert_same_consensus(want, h.fetch(), f"round {rnd}")
                assert np.array_equal(h.votes(), want["votes"])
            for e, b in zip(ext, before):
                assert e is buf or torch.equal(e, b)
        assert h.stats()["graph_rounds"] == 10
