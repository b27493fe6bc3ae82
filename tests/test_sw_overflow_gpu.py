"""Pairs whose scores pass 16 bits beside pairs whose scores do not.

Two pairs share the words of the throughput forms.  One that runs past 65,535
wraps and, at large gap costs, leaves a value below the gap cost in one cell;
the pair beside it must not notice.  Here that pair opens a gap in exactly
that cell: in the by-pair form (batches above 4,096 pairs) against the
oracle, and among the hits of one query (profile shared, stripes) against
the score its alignment has by construction."""
import numpy as np
import pytest

import oracle
from sa_util import make_db
from topaz_b200 import alphabet as ab, native, synth

pytestmark = pytest.mark.gpu


def _gapped(rng, q, row, col, ns, filler, span, horizontal):
    """Subject that follows q up to (row, col), opens a gap there and goes on."""
    s = rng.choice(filler, ns).astype(np.int8)
    before = min(span, row + 1, col + 1)
    s[col + 1 - before:col + 1] = q[row + 1 - before:row + 1]
    at, r = (col + 2, row + 1) if horizontal else (col + 1, row + 2)
    after = min(span, len(q) - r, ns - at)
    s[at:at + after] = q[r:r + after]
    return s


# rows, columns, gap costs, and the cell where the pair of one letter leaves
# a value below gap_open
@pytest.mark.parametrize("nq,ns,go,ge,row,col", [(600, 1000, 255, 254, 511, 767),
                                                 (1024, 1500, 200, 150, 512, 946),
                                                 (1024, 1500, 100, 90, 515, 1240)])
def test_by_pair(cuda, nq, ns, go, ge, row, col):
    torch = cuda
    rng = np.random.default_rng(go)
    mat = np.full((25, 25), -4, np.int8)
    np.fill_diagonal(mat, 127)
    q = rng.integers(0, 17, nq).astype(np.int8)
    kinds = [(np.full(nq, 17, np.int8), np.full(ns, 17, np.int8))]
    kinds += [(q, _gapped(rng, q, row, col, ns, np.arange(18, 25), 64, h)) for h in (False, True)]
    kinds.insert(2, kinds[0])                       # every second pair overflows
    ql = np.array([nq] * 4, np.int32)
    sl = np.array([ns] * 4, np.int32)
    qc, sc = np.concatenate([k[0] for k in kinds]), np.concatenate([k[1] for k in kinds])
    off4, soff4 = np.arange(4, dtype=np.int64) * nq, np.arange(4, dtype=np.int64) * ns
    want = np.stack(oracle.oracle_sw(qc, off4, ql, sc, soff4, sl, mat, go, ge))
    assert list(want[3]) == [native.TPZ_SW_DROPPED, 0, native.TPZ_SW_DROPPED, 0]
    assert (want[1:3, [1, 3]] > [[col], [row]]).all()           # their paths pass the cell
    n = 4 * 1100
    pick = np.arange(n) % 4
    t = {"q": qc, "qoff": off4[pick], "qlen": ql[pick], "s": sc, "soff": soff4[pick], "slen": sl[pick]}
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in t.items()}
    for k in ("score", "ref_end", "read_end", "status"):
        t[k] = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    native.sw_batch_torch(t, mat, go, ge)
    got = np.stack([t[k].cpu().numpy() for k in ("score", "ref_end", "read_end", "status")])
    bad = np.flatnonzero((got != want[:, pick]).any(axis=0))
    assert bad.size == 0, (bad.size, got[:, bad[:4]], want[:, pick[bad[:4]]])


@pytest.mark.parametrize("report", [True, False])
def test_hits_of_one_query(cuda, report):
    # letters: the query has 0-11; a subject of 12-19 scores 17 against every
    # row of it, so its columns are alike and row 3841 (17 * 3842 + 238 is the
    # first past 65,535) wraps in all of them; 20-23 match nothing
    rng = np.random.default_rng(5)
    go, ge, row, col, nq, span = 60, 50, 3841, 5150, 8192, 300
    mat = np.full((25, 25), -128, np.int8)
    mat[:20, :20] = 17
    mat[:12, :12] = -128
    np.fill_diagonal(mat[:12, :12], 17)
    q = rng.integers(0, 12, nq).astype(np.int8)
    seqs, paired = [], 8
    for k in range(paired):                          # sorted by length they alternate
        high = rng.integers(12, 20, 6000 - 2 * k).astype(np.int8)
        high[-30:] = q[1000:1030]                    # something to find it by
        seqs += [high, _gapped(rng, q, row, col, 5999 - 2 * k, np.arange(20, 24), span, False)]
    order = np.frombuffer(ab.MATRIX_ORDER.encode(), np.uint8)
    db = make_db(synth.Proteins(["p%d" % i for i in range(len(seqs))], [order[x] for x in seqs]))
    kw = {"report": {"max_evalue": 1e30}} if report else {}
    r = native.Index(db).search([ab.aa_to_internal(order[q]).tobytes()], mat, gap_open=go, gap_extend=ge, **kw)
    got = {int(p): [int(r[k][i]) for k in ("rawscore", "qend", "send", "sw_status")]
           for i, p in enumerate(r["protein"])}
    if not report:                                   # dropped pairs are not reported
        assert [got.pop(p)[3] for p in range(0, 2 * paired, 2)] == [native.TPZ_SW_DROPPED] * paired
    want = [17 * 2 * span - go, row + 1 + span, col + span, native.TPZ_SW_OK]
    first = [int(x[0]) for x in oracle.oracle_sw(q, np.zeros(1, np.int64), np.array([nq], np.int32), seqs[1],
                                                 np.zeros(1, np.int64), np.array([len(seqs[1])], np.int32),
                                                 mat, go, ge)]
    assert [first[0], first[2], first[1], first[3]] == want
    assert got == {p: want for p in range(1, 2 * paired, 2)}
