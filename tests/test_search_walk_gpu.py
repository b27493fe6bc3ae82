"""The walk and the hitlist where their parallel forms have edges: runs of
pops that cross blocks of chain elements (rows 8, 32, 64, ... on), rises of
hits already listed, capacities around a batch of 32 pops, evictions at one
and over several scores, stops at -S inside a batch, and cursor counts of
every shared-memory class up to the one that spills -- pop by pop against
the oracle, with the hits' Smith-Waterman columns, on a database of protein
families (long runs of similar rows); and the extensions they rest on, at
every kind of end."""
import numpy as np
import pytest

import oracle
from sa_util import make_db
from topaz_b200 import alphabet as ab, native, synth

pytestmark = pytest.mark.gpu

BLOSUM62 = synth.matrix("BLOSUM62")


@pytest.fixture(scope="module")
def family_db():
    rng = np.random.Generator(np.random.PCG64(71))
    prot = synth.protein_db(1200, seed=70)
    seqs = list(prot.seqs)
    members = []
    for f in range(12):
        base = synth.random_residues(rng, int(rng.integers(60, 500)))
        for identity in rng.uniform(0.5, 1.0, 90):
            members.append(synth.mutate(rng, base, float(identity), indel_rate=0.01))
        # proteins that repeat a piece of the family: one protein, many rows
        members += [np.concatenate([synth.mutate(rng, base[:60], 0.8) for _ in range(6)]) for _ in range(20)]
    seqs += members
    order = rng.permutation(len(seqs))
    db = make_db(synth.Proteins(["p%d" % i for i in range(len(seqs))], [seqs[i] for i in order]))
    qs = [members[i] for i in rng.choice(len(members), 10, replace=False)]
    qs += [synth.random_residues(rng, n) for n in (5, 6, 7, 37, 260, 261, 600)]
    # capacity 1.5 * num_hits above 3000 residues; two cursors per searched
    # position: classes of 512, 1,024, 2,048 (600 residues above), 3,072 (1,300)
    # and 5,600 (1,700 and more), in global memory above 2,805
    qs += [synth.random_residues(rng, 1300),
           np.concatenate([members[3], synth.random_residues(rng, 1700)]),
           np.concatenate([synth.random_residues(rng, 3000), members[40]]),
           np.concatenate([synth.random_residues(rng, 4500), members[200]])]
    return db, [ab.aa_to_internal(s).tobytes() for s in qs]


@pytest.mark.parametrize("seeds,aligns,num_hits", [(300000, 5000, 100), (300000, 300, 40), (300000, 33, 1),
                                                   (300000, 32, 21), (300000, 31, 2), (300000, 1, 3),
                                                   (300000, 64, 10), (1, 5000, 100), (33, 5, 100), (777, 64, 10)])
def test_every_pop_and_hit(cuda, family_db, seeds, aligns, num_hits):
    db, qs = family_db
    ix = native.Index(db)
    cap = 1 << 17
    r = ix.search(qs, BLOSUM62, num_hits=num_hits, seeds=seeds, alignments=aligns, trace_pops=cap)
    opts = oracle.Opts(num_hits, 1e-3, 11, 1, 0.267, 0.041, 0.14, 5, seeds, aligns)
    longest = 0
    for q, qi in enumerate(qs):
        P, hits, npops, ncnt, nh = oracle.oracle_query(db, qi, BLOSUM62, opts)
        assert nh >= 0 and npops <= cap
        assert (r["npops"][q], r["ncounted"][q]) == (npops, ncnt), q
        for name in ("row", "off", "score", "len", "counted"):
            assert (r["trace_" + name][q, :npops] == P[name][:npops]).all(), (q, name)
        a, b = r["hit_off"][q], r["hit_off"][q + 1]
        assert list(r["protein"][a:b]) == [h.db_index for h in hits]
        assert list(r["gapless_score"][a:b]) == [h.gapless_score for h in hits]
        assert list(r["gapless_length"][a:b]) == [h.gapless_length for h in hits]
        assert list(r["suffix_offset"][a:b]) == [h.suffix_offset for h in hits]
        on = [i for i, h in enumerate(hits) if h.gapless_score >= 40]
        for ours, name in (("sw_status", "status"), ("rawscore", "rawscore"), ("qend", "qend"), ("send", "send")):
            assert [int(r[ours][a + i]) for i in on] == [getattr(hits[i], name) for i in on], (q, name)
        longest = max(longest, npops)
    if seeds == 300000:
        assert r["refill_elems"] > 0 and longest > 2000


@pytest.mark.parametrize("name,scale", [("BLOSUM62", 1), ("PAM30", 1), ("BLOSUM62", 11)])
def test_extensions_at_every_end(cuda, family_db, name, scale):
    # window ends at the query's start and end, the text's start and end,
    # protein ends, 32-byte rounds and the 128-residue limit; entries up to 121
    db, qs = family_db
    mat = (synth.matrix(name).astype(np.int64) * scale).astype(np.int8)
    ix, orc = native.Index(db), oracle.liboracle()
    rng = np.random.default_rng(3)
    first = [int(np.flatnonzero(db.SA == p)[0]) for p in (0, 1, 31, 32, 33, db.Tsize - 2, db.Tsize - 34)]
    qof, off, row = [], [], []
    for qi, q in enumerate(qs):
        ends = [i for i in (0, 1, 2, 31, 32, 33, 34, 127, 128, 129, len(q) // 2) if i < len(q)]
        ends += [len(q) - 1 - i for i in (0, 1, 31, 32, 33, 127, 128) if i < len(q)]
        for i in ends:
            near = ix.sa_search([q[i:]])[0]
            rows = first + [min(max(int(near) + d, 0), db.Tsize - 1) for d in (-2, -1, 0, 1)]
            rows += rng.integers(0, db.Tsize, 3).tolist()
            for r in rows:
                qof.append(qi)
                off.append(i)
                row.append(r)
    sc, ln = ix.sa_hsp(qs, qof, off, row, mat)
    sub = ab.internal_to_index(np.arange(65, 90, dtype=np.uint8)).astype(np.int64)
    for k in range(len(row)):
        want = _extension(db.T, int(db.SA[row[k]]), qs[qof[k]], off[k], mat, sub)
        assert (sc[k], ln[k]) == want, (qof[k], off[k], row[k])


def _extension(T, at, q, off, mat, sub):
    """sa_hsp of one pair of positions, residue by residue."""
    if T[at] != q[off]:
        return 0, -1

    def walk(steps, first):
        run = best = arg = 0
        for i in range(first, steps):
            t, c = (T[at + i], q[off + i]) if first == 0 else (T[at - i], q[off - i])
            if t == 10:
                break
            run += int(mat[sub[t - 65], sub[c - 65]])
            if run >= best:
                best, arg = run, i
        return best, arg

    r, i = walk(min(len(T) - at, len(q) - off, 128), 0)
    l, j = walk(min(at, off, 128), 1)
    return r + l, i + j
