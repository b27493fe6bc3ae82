"""Where the batch call changes its form: the lanes per pair, rows per lane
and warps per pair at the ends of each query-length class, the batch size at
which the stripe form hands over, long subjects through the letter and
boundary rings, and scores around the 16-bit drop -- against the oracle, and
the same pairs in another batch against themselves."""
import numpy as np
import pytest

import oracle
from topaz_b200 import native, synth

pytestmark = pytest.mark.gpu

EDGES = (1, 2, 16, 17, 32, 33, 36, 64, 65, 72, 128, 129, 144, 256, 257, 288, 289, 384, 385, 511, 512, 513, 768, 992,
         1023, 1024, 1025, 1280, 2047, 2048, 2049, 4095, 4096, 4097, 6144, 8192)


def _pairs(qs, ss):
    ql = np.array([len(x) for x in qs], np.int32)
    sl = np.array([len(x) for x in ss], np.int32)
    return synth.PairSet(np.concatenate(qs), (np.cumsum(ql) - ql).astype(np.int64), ql,
                         np.concatenate(ss + [np.zeros(1, np.int8)]),
                         (np.cumsum(sl) - sl).astype(np.int64), sl, 0)


def _run(torch, ps, mat, go, ge):
    t = {k: torch.from_numpy(np.ascontiguousarray(getattr(ps, k))).cuda()
         for k in ("q", "qoff", "qlen", "s", "soff", "slen")}
    for k in ("score", "ref_end", "read_end", "status"):
        t[k] = torch.full((ps.n,), -7, dtype=torch.int32, device="cuda")
    native.sw_batch_torch(t, mat, go, ge)
    torch.cuda.synchronize()
    return np.stack([t[k].cpu().numpy() for k in ("score", "ref_end", "read_end", "status")])


def _edge_pairs(rng):
    qs, ss = [], []
    for n in EDGES:
        q = rng.integers(0, 25, n).astype(np.int8)
        for m in (0, 1, 63, 64, 65, 129, 700):
            s = rng.integers(0, 25, m).astype(np.int8)
            k = min(n, m) // 2
            at = int(rng.integers(0, m - k + 1)) if m else 0
            s[at:at + k] = q[n - k:]               # an end of the query, across stripes
            qs.append(q)
            ss.append(s)
    return qs, ss


@pytest.mark.parametrize("name,go,ge,small", [("BLOSUM62", 11, 1, True), ("BLOSUM62", 11, 1, False),
                                              ("PAM250", 1, 0, False), ("BLOSUM45", 255, 254, True)])
def test_class_edges(cuda, name, go, ge, small):
    qs, ss = _edge_pairs(np.random.default_rng(go + 7 * small))
    n = len(qs)
    if not small:                                   # past the size where short queries change form
        fill = synth.sw_pairs(4097, seed=go, q_range=(1, 90), q_median=30, s_range=(0, 200), s_median=60)
        qs += [fill.q[o:o + k] for o, k in zip(fill.qoff, fill.qlen)]
        ss += [fill.s[o:o + k] for o, k in zip(fill.soff, fill.slen)]
    ps, mat = _pairs(qs, ss), synth.matrix(name)
    assert (ps.n > 4096) != small and n <= 4096
    got = _run(cuda, ps, mat, go, ge)
    want = np.stack(oracle.oracle_sw(ps.q, ps.qoff, ps.qlen, ps.s, ps.soff, ps.slen, mat, go, ge))
    bad = np.flatnonzero((got != want).any(axis=0))
    assert bad.size == 0, (bad[:5], got[:, bad[:5]], want[:, bad[:5]], ps.qlen[bad[:5]], ps.slen[bad[:5]])


@pytest.mark.parametrize("n", [1, 3, 1025, 4095, 4096, 4097])
def test_batch_size_where_the_form_changes(cuda, n):
    ps = synth.sw_pairs(n, seed=n, s_range=(0, 3000))
    mat = synth.matrix("BLOSUM62")
    got = _run(cuda, ps, mat, 11, 1)
    want = np.stack(oracle.oracle_sw(ps.q, ps.qoff, ps.qlen, ps.s, ps.soff, ps.slen, mat))
    assert (got == want).all()


@pytest.mark.parametrize("n", [300, 1536, 1537, 4096, 4097, 8192, 8193])
def test_class_edges_at_every_batch_size(cuda, n):
    # the ends of the length classes again, in the forms that a batch of n takes
    qs, ss = _edge_pairs(np.random.default_rng(n))
    rng = np.random.default_rng(n + 1)
    for k in (17, 64, 65, 128, 129, 256, 257):      # both sides of the subject length in the rule
        for m in (3071, 3072):
            q = rng.integers(0, 25, k).astype(np.int8)
            s = rng.integers(0, 25, m).astype(np.int8)
            s[-k:] = q
            qs.append(q)
            ss.append(s)
    fill = synth.sw_pairs(n - len(qs), seed=n, q_range=(1, 300), q_median=60, s_range=(0, 200), s_median=60)
    qs += [fill.q[o:o + k] for o, k in zip(fill.qoff, fill.qlen)]
    ss += [fill.s[o:o + k] for o, k in zip(fill.soff, fill.slen)]
    ps, mat = _pairs(qs, ss), synth.matrix("BLOSUM62")
    assert ps.n == n
    got = _run(cuda, ps, mat, 11, 1)
    want = np.stack(oracle.oracle_sw(ps.q, ps.qoff, ps.qlen, ps.s, ps.soff, ps.slen, mat))
    bad = np.flatnonzero((got != want).any(axis=0))
    assert bad.size == 0, (bad[:5], got[:, bad[:5]], want[:, bad[:5]], ps.qlen[bad[:5]], ps.slen[bad[:5]])


def test_drop_at_16_bits_in_every_form(cuda):
    # runs of one letter scoring 127 each: 258 of them make 32766, 259 are
    # dropped; next to pairs of the same tasks that are not
    mat = synth.matrix("BLOSUM62").copy()
    mat[17, 17] = 127
    qs, ss = [], []
    for n in (257, 258, 259, 300, 600, 1024, 1025, 3000):
        for m in (258, 259, 1000):
            qs.append(np.full(n, 17, np.int8))
            ss.append(np.full(m, 17, np.int8))
            qs.append(np.full(n, 16, np.int8))
            ss.append(np.full(m, 16, np.int8))
    for copies in (1, 90):                          # stripe form, throughput form
        ps = _pairs(qs * copies, ss * copies)
        got = _run(cuda, ps, mat, 11, 1)
        want = np.stack(oracle.oracle_sw(ps.q, ps.qoff, ps.qlen, ps.s, ps.soff, ps.slen, mat))
        assert (want[3] == native.TPZ_SW_DROPPED).any() and (want[0] == 32766).any()
        bad = np.flatnonzero((got != want).any(axis=0))
        assert bad.size == 0, (bad[:5], got[:, bad[:5]], want[:, bad[:5]], ps.qlen[bad[:5]])
