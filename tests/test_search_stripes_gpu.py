"""The query-major Smith-Waterman kernels at the query lengths where stripes
begin (one, two, ... eight of them, and each class of stripe counts), with
16 to more than 256 pairs of a query, so that pair lists are cut: scores and
ends (all hits) and scores alone (report mode) against the by-pair batch,
which the oracle pins, and the oracle itself on a sample."""
import numpy as np
import pytest

import oracle
from sa_util import make_db
from topaz_b200 import alphabet as ab, native, synth

pytestmark = pytest.mark.gpu

MAT = synth.matrix("BLOSUM62")


@pytest.fixture(scope="module")
def db_and_families():
    rng = np.random.Generator(np.random.PCG64(93))
    bases = [synth.random_residues(rng, n) for n in (180, 260, 90, 400)]
    members = [[synth.mutate(rng, b, float(i), indel_rate=0.01) for i in rng.uniform(0.6, 0.95, n)]
               for b, n in zip(bases, (20, 130, 120, 110))]
    seqs = [m for fam in members for m in fam] + list(synth.protein_db(200, seed=94).seqs)
    return make_db(synth.Proteins(["p%d" % i for i in range(len(seqs))], seqs)), bases


# (length, families in it): 20 pairs, or up to 380 of them
QUERIES = [(n, f) for n in (40, 64, 65, 128, 256, 257, 512, 1000, 1024, 1025, 1300, 2048, 2049, 3073, 4097, 5000,
                            5121, 6145, 7169, 8192) for f in ((0,), (0, 1, 2, 3))]


def _query(rng, n, fams, bases):
    q = synth.random_residues(rng, n)
    room = n // len(fams)
    for k, f in enumerate(fams):                     # a piece in each part, at its end
        piece = synth.mutate(rng, bases[f], 0.9)[-room:]
        q[(k + 1) * room - len(piece):(k + 1) * room] = piece
    return q


@pytest.fixture(scope="module")
def searched(db_and_families):
    db, bases = db_and_families
    rng = np.random.Generator(np.random.PCG64(95))
    qs = [ab.aa_to_internal(_query(rng, n, f, bases)) for n, f in QUERIES]
    ix = native.Index(db)
    return db, ix, qs, ix.search([q.tobytes() for q in qs], MAT, num_hits=400)


def _subjects(db, proteins):
    ps, pl = db.pstart, db.ind["protein_len"]
    return [ab.internal_to_index(db.T[ps[p]:ps[p] + pl[p]]) for p in proteins]


def _pairs(db, q, proteins):
    qi, ss = ab.internal_to_index(q), _subjects(db, proteins)
    sl = np.array([len(s) for s in ss], np.int32)
    n = len(ss)
    return (qi, np.zeros(n, np.int64), np.full(n, len(qi), np.int32), np.concatenate(ss),
            (np.cumsum(sl) - sl).astype(np.int64), sl)


def test_scores_and_ends(cuda, searched):
    db, _, qs, r = searched
    rng = np.random.default_rng(3)
    counts = []
    for k, q in enumerate(qs):
        sel = np.arange(r["hit_off"][k], r["hit_off"][k + 1])
        sel = sel[r["sw_status"][sel] == native.TPZ_SW_OK]
        counts.append(len(sel))
        got = np.stack([r[f][sel] for f in ("rawscore", "send", "qend")])
        want = np.stack(native.sw_batch_host(*_pairs(db, q, r["protein"][sel]), MAT)[:3])
        assert (got == want).all(), QUERIES[k]
        pick = rng.choice(len(sel), min(len(sel), 12), replace=False)
        want = np.stack(oracle.oracle_sw(*_pairs(db, q, r["protein"][sel[pick]]), MAT)[:3])
        assert (got[:, pick] == want).all(), QUERIES[k]
    striped = [c for c, (n, _) in zip(counts, QUERIES) if n > 1024]
    assert sum(c >= 16 for c in counts) > len(counts) - 6 and max(striped) > 256 and min(striped) >= 16


def test_scores_alone_rank_the_hits(cuda, searched):
    db, ix, qs, r = searched
    top = ix.search([q.tobytes() for q in qs], MAT, num_hits=400, report={"max_evalue": 1e30})
    for k in range(len(qs)):
        a, b = r["hit_off"][k], r["hit_off"][k + 1]
        raw = np.where(r["sw_status"][a:b] == native.TPZ_SW_OK, r["rawscore"][a:b], -1)
        order = np.argsort(-raw, kind="stable")
        order = order[raw[order] >= 0][:400]
        c = top["hit_off"][k]
        n = int((top["sw_status"][c:top["hit_off"][k + 1]] == native.TPZ_SW_OK).sum())
        assert n == len(order)
        assert list(top["protein"][c:c + n]) == list(r["protein"][a:b][order]), QUERIES[k]
        assert list(top["rawscore"][c:c + n]) == list(raw[order]), QUERIES[k]
