"""Timed cases of the search path, through the calls a user's program makes.

Kinds of work, each over its range of sizes:

  sw_device   batched Smith-Waterman of (query, subject) pairs that sit in
              device memory (native.sw_batch_torch)
  sw_host     the same from host buffers, copies included
              (native.sw_batch_host)
  search      whole queries against a resident database: seed lookup,
              extension, walk, Smith-Waterman of the hits, ranking
              (native.Index.search)
  extend      gapless extensions of (query, offset, suffix-array row) triples
              (native.Index.sa_hsp)
  index       the suffix array of a database text (native.sa_build)

Residues follow the Robinson-Robinson background; homologues are mutated
with BLOSUM62-conditional substitutions and short indels; lengths are
log-normal (sigma 0.6) clipped to the stated range.  Every result is an
integer, or a double computed from one, so all comparisons are exact.
"""
import math

import numpy as np
import torch

from topaz_b200 import alphabet, dbformat, native, synth

DEV = "cuda"
SIGMA = 0.6

# ------------------------------------------------------------------- cases


def listed():
    return [
        # one user's handful of pairs: launches and latency
        _sw("sw_64_pairs", 64),
        # the reported hits of one search batch re-aligned for their ends
        _sw("sw_20k_pairs", 20_000),
        # all-against-all scoring: the batched microbench's pairs
        _sw("sw_200k_pairs", 200_000),
        # peptides and domain fragments under a short-query matrix
        _sw("sw_100k_short_pam30", 100_000, q_median=60, q_lo=8, q_hi=150, s_median=150, s_lo=0,
            s_hi=1500, matrix="PAM30", gap_open=9, gap_extend=1),
        # multi-domain proteins, longer than one stripe of the query
        _sw("sw_1500_long", 1_500, q_median=2500, q_lo=1025, q_hi=8192, s_median=1200, s_lo=200,
            s_hi=5000),
        # a host program's pairs: host buffers in, host results out
        _sw("sw_host_80k", 80_000, kind="sw_host"),
        # an interactive search: one query, default sensitivity
        _search("search_one_query", 1, 50_000),
        # a serving loop's request
        _search("search_40_queries", 40, 50_000),
        # batch search at default sensitivity, ranked and cut on the device
        _search("search_1000_queries", 1_000, 150_000),
        # --fast --blasttab on FASTA residues: SEG and statistics on the device
        _search("search_fast_blasttab", 500, 100_000, ingest=1, stats=True, seeds=100_000,
                alignments=1_500),
        # every hit of long queries with its end coordinates, another matrix
        _search("search_all_hits_long", 48, 50_000, q_median=1100, q_lo=300, q_hi=4000,
                report=False, matrix="BLOSUM45", gap_open=14, gap_extend=2),
        # the index of a new database
        {"name": "index_20k_proteins", "kind": "index", "proteins": 20_000},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["sw_device", "sw_device", "sw_long", "sw_short", "sw_host", "search",
                       "search", "search_long", "extend", "index"])
    matrix, go, ge = rng.choice([("BLOSUM62", 11, 1), ("BLOSUM62", 11, 1), ("BLOSUM50", 13, 2),
                                 ("BLOSUM80", 10, 1), ("PAM250", 14, 2)])
    opts = {"matrix": matrix, "gap_open": go, "gap_extend": ge}
    if kind == "sw_device":
        return _sw(None, logint(1, 120_000), homologs=rng.choice([0.05, 0.2, 0.6]), **opts)
    if kind == "sw_long":
        return _sw(None, logint(2, 1_200), q_median=2500, q_lo=1025, q_hi=8192, s_median=1200,
                   s_lo=200, s_hi=5000, **opts)
    if kind == "sw_short":
        return _sw(None, logint(10, 100_000), q_median=60, q_lo=1, q_hi=150, s_median=150, s_lo=0,
                   s_hi=1500, matrix="PAM30", gap_open=9, gap_extend=1)
    if kind == "sw_host":
        return _sw(None, logint(3, 80_000), kind="sw_host", **opts)
    if kind == "extend":
        return {"kind": "extend", "proteins": logint(500, 50_000), "queries": logint(1, 500),
                "triples": logint(100, 500_000), "matrix": matrix}
    if kind == "index":
        return {"kind": "index", "proteins": logint(200, 40_000)}
    fast = rng.random() < 0.4
    long_q = kind == "search_long"
    form = rng.choice(["report", "stats", "all"] if long_q else ["report", "report", "stats"])
    return _search(None, logint(1, 40 if long_q else 500), logint(2_000, 120_000),
                   q_median=1100 if long_q else 300, q_lo=300 if long_q else 30,
                   q_hi=4000 if long_q else 1500, report=form != "all", stats=form == "stats",
                   ingest=rng.choice([0, 1, 2]), seeds=100_000 if fast else 300_000,
                   alignments=1_500 if fast else 5_000, **opts)


def _sw(name, n, kind="sw_device", q_median=350, q_lo=30, q_hi=1000, s_median=350, s_lo=30,
        s_hi=5000, homologs=0.2, matrix="BLOSUM62", gap_open=11, gap_extend=1):
    c = {"kind": kind, "pairs": n, "q_median": q_median, "q_lo": q_lo, "q_hi": q_hi,
         "s_median": s_median, "s_lo": s_lo, "s_hi": s_hi, "homologs": homologs, "matrix": matrix,
         "gap_open": gap_open, "gap_extend": gap_extend}
    return c if name is None else {"name": name, **c}


def _search(name, queries, proteins, q_median=300, q_lo=50, q_hi=1500, report=True, stats=False,
            ingest=0, seeds=300_000, alignments=5_000, matrix="BLOSUM62", gap_open=11,
            gap_extend=1):
    c = {"kind": "search", "queries": queries, "proteins": proteins, "q_median": q_median,
         "q_lo": q_lo, "q_hi": q_hi, "report": report, "stats": stats, "ingest": ingest,
         "seeds": seeds, "alignments": alignments, "matrix": matrix, "gap_open": gap_open,
         "gap_extend": gap_extend}
    return c if name is None else {"name": name, **c}


# ----------------------------------------------------------------- residues
# amino acids are numbered 0..19 in the order of synth.AA20 until they are
# mapped to matrix indices, internal letters or upper-case residues


def _table(values):
    return torch.from_numpy(np.array(values)).to(DEV)


def _draw_table(p):
    """65,536 amino-acid numbers in the proportions p."""
    cum = np.rint(np.cumsum(p) / np.sum(p) * 65536).astype(np.int64)
    return np.searchsorted(cum, np.arange(65536), side="right").astype(np.uint8)


def _substitutes():
    """Per amino acid: 65,536 draws of what replaces it."""
    idx = alphabet.aa_to_index(synth.AA20).astype(np.int64)
    s = synth.matrix("BLOSUM62")[np.ix_(idx, idx)].astype(np.float64)
    p = synth.P20 * np.exp(0.32 * s)
    np.fill_diagonal(p, 0.0)
    return np.stack([_draw_table(row) for row in p])


class _Draw:
    """Seeded random residues and lengths on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)
        self.background = _table(_draw_table(synth.P20))
        self.sub = _table(_substitutes())

    def ints(self, hi, n):
        return torch.randint(0, hi, (n,), generator=self.g, device=DEV)

    def unit(self, n):
        return torch.rand(n, generator=self.g, device=DEV)

    def residues(self, n):
        return self.background[self.ints(65536, n)]

    def lengths(self, n, median, lo, hi):
        z = torch.randn(n, generator=self.g, device=DEV, dtype=torch.float64)
        x = torch.round(torch.exp(math.log(median) + SIGMA * z))
        return x.clamp(lo, hi).to(torch.int64)

    def mutated(self, src, start, seg, identity):
        """The residues at src[start + k], segment by segment (seg: the
        segment of each), substituted with probability 1 - identity[seg];
        at 2 % of the positions a short insertion or deletion shifts what
        follows in the segment."""
        n = len(seg)
        step = torch.where(self.unit(n) < 0.5, 1, -1) * (1 + self.ints(3, n))
        shift = torch.cumsum(torch.where(self.unit(n) < 0.02, step, 0), 0)
        first = torch.searchsorted(seg, seg)
        at = (start + shift - shift[first]).clamp(0, len(src) - 1)
        r = src[at]
        other = self.sub[r.long(), self.ints(65536, n)]
        return torch.where(self.unit(n) < identity[seg], r, other)


def _offsets(lens):
    return torch.cumsum(lens, 0) - lens


def _positions(lens):
    """(segment, index in it) of every position of consecutive segments."""
    seg = torch.repeat_interleave(torch.arange(len(lens), device=DEV), lens)
    return seg, torch.arange(len(seg), device=DEV) - _offsets(lens)[seg]


def _pairs(case, seed):
    """Pairs in matrix indices: a share of the subjects are homologues of
    their query at 25-60 % identity, centred in background residues."""
    d = _Draw(seed)
    n = case["pairs"]
    ql = d.lengths(n, case["q_median"], case["q_lo"], case["q_hi"])
    sl = d.lengths(n, case["s_median"], case["s_lo"], case["s_hi"])
    hom = d.unit(n) < case["homologs"]
    sl = torch.where(hom, torch.maximum(sl, ql.clamp(max=case["s_hi"])), sl)
    q = d.residues(int(ql.sum()))
    qo, so = _offsets(ql), _offsets(sl)
    seg, k = _positions(sl)
    core = k - torch.div(sl - torch.minimum(sl, ql), 2, rounding_mode="floor")[seg]
    inside = hom[seg] & (core >= 0) & (core < ql[seg])
    s = d.residues(len(seg))
    at = torch.nonzero(inside).squeeze(1)
    if len(at):
        identity = 0.25 + 0.35 * d.unit(n)
        s[at] = d.mutated(q, qo[seg[at]] + core[at], seg[at], identity)
    idx = _table(alphabet.aa_to_index(synth.AA20).astype(np.int8))
    pad = torch.zeros(1, dtype=torch.int8, device=DEV)
    return {"q": torch.cat([idx[q.long()], pad]), "qoff": qo, "qlen": ql.to(torch.int32),
            "s": torch.cat([idx[s.long()], pad]), "soff": so, "slen": sl.to(torch.int32)}


def _database(proteins, seed):
    """(amino-acid numbers of all proteins, their lengths and offsets, the
    database without its suffix array); proteins of 50-2000 residues."""
    # the lengths belong to the case, so its text has one size for every seed
    lens = _Draw(proteins).lengths(proteins, 300, 50, 2000)
    d = _Draw(seed)
    res = d.residues(int(lens.sum()))
    off = _offsets(lens)
    seg, k = _positions(lens)
    text = torch.full((len(res) + proteins,), 10, dtype=torch.uint8, device=DEV)
    text[off[seg] + seg + k] = _table(alphabet.aa_to_internal(synth.AA20))[res.long()]
    ind = np.zeros(proteins, dtype=dbformat.IND_DTYPE)
    head = np.array([len("db%d" % i) for i in range(proteins)], np.int64)
    ind["header_start"] = np.cumsum(head + 1) - (head + 1)
    ind["header_len"] = head
    ind["protein_start"] = (off + torch.arange(proteins, device=DEV)).cpu().numpy()
    ind["protein_len"] = lens.cpu().numpy()
    headers = b"".join(b"db%d\n" % i for i in range(proteins))
    return res, lens, off, dbformat.Database(text.cpu().numpy(), None, ind, headers)


def _queries(d, n, median, lo, hi, res, lens, off, letters):
    """n queries as bytes: half mutated from database proteins at 30-90 %
    identity, half background; one in twenty has a low-complexity tract."""
    ql = d.lengths(n, median, lo, hi)
    pick = d.ints(len(lens), n)
    seg, k = _positions(ql)
    own = (d.unit(n) < 0.5)[seg] & (k < lens[pick][seg])
    r = d.residues(len(seg))
    at = torch.nonzero(own).squeeze(1)
    if len(at):
        identity = 0.30 + 0.60 * d.unit(n)
        r[at] = d.mutated(res, off[pick][seg[at]] + k[at], seg[at], identity)
    tract = (d.unit(n) < 0.05)[seg] & (k >= 20) & (k < 36)
    r = torch.where(tract, (seg % 20).to(torch.uint8), r)
    b = _table(letters)[r.long()].cpu().numpy().tobytes()
    o, ln = _offsets(ql).tolist(), ql.tolist()
    return [b[x:x + y] for x, y in zip(o, ln)]


def _index(case, seed):
    res, lens, off, db = _database(case["proteins"], seed)
    db.SA = native.sa_build(db.T)
    return res, lens, off, native.Index(db)


# ------------------------------------------------------------------ running


def prepare(case, seed):
    kind = case["kind"]
    if kind == "index":
        return {"kind": kind, "T": _database(case["proteins"], seed)[3].T}
    state = {"kind": kind, "mat": native.matrix(case["matrix"])}
    if kind in ("sw_device", "sw_host"):
        t = _pairs(case, seed)
        if kind == "sw_device":
            for name in ("score", "ref_end", "read_end", "status"):
                t[name] = torch.zeros(case["pairs"], dtype=torch.int32, device=DEV)
        else:
            t = {name: x.cpu().pin_memory().numpy() for name, x in t.items()}
        state.update(t=t, go=case["gap_open"], ge=case["gap_extend"])
        return state
    res, lens, off, ix = _index(case, seed)
    d = _Draw(seed + 1_000_003)
    if kind == "extend":
        # offsets and rows as a seeding loop meets them: the rows around the
        # lower bound of the query's words
        qs = _queries(d, case["queries"], 300, 50, 1500, res, lens, off,
                      alphabet.aa_to_internal(synth.AA20))
        n = case["triples"]
        query = d.ints(len(qs), n).cpu().numpy()
        at = (d.unit(n).cpu().numpy() * (np.array([len(q) for q in qs])[query] - 6)).astype(np.int32)
        bound = ix.sa_search([qs[q][a:] for q, a in zip(query.tolist(), at.tolist())])
        row = np.clip(bound + d.ints(64, n).cpu().numpy() - 32, 0, len(ix.db.SA) - 1)
        state.update(ix=ix, queries=qs, query=query.astype(np.int32), at=at, row=row)
        return state
    letters = synth.AA20 if case["ingest"] else alphabet.aa_to_internal(synth.AA20)
    qs = _queries(d, case["queries"], case["q_median"], case["q_lo"], case["q_hi"], res, lens, off,
                  letters)
    report = {"max_evalue": 1e-3, "stats": case["stats"]} if case["report"] else None
    width = 100 if case["report"] else case["alignments"]
    state.update(ix=ix, queries=qs, width=width, opts={
        "gap_open": case["gap_open"], "gap_extend": case["gap_extend"], "seeds": case["seeds"],
        "alignments": case["alignments"], "report": report, "ingest": case["ingest"]})
    return state


# what search returns besides its own timings and counts of internal work
_PER_QUERY = ("npops", "ncounted", "status")
_PER_HIT = ("protein", "gapless_score", "gapless_length", "suffix_offset", "rawscore", "qend",
            "send", "sw_status", "bitscore", "evalue", "qstart", "sstart", "length", "gapopen",
            "mismatch", "identity")


def _hit_tables(out, width):
    """A row of `width` places per query for each column of its hits."""
    off = out["hit_off"]
    count = np.diff(off)
    query = np.repeat(np.arange(len(count)), count)
    place = np.arange(len(query)) - np.repeat(off[:-1], count)
    tables = {"hits": count}
    for name in _PER_HIT:
        if name in out:
            real = name in ("bitscore", "evalue", "identity")
            tables[name] = np.full((len(count), width), -1, np.float64 if real else np.int32)
            tables[name][query, place] = out[name]
    return tables


def run(state):
    kind = state["kind"]
    if kind == "index":
        return native.sa_build(state["T"])
    if kind == "sw_device":
        t = state["t"]
        native.sw_batch_torch(t, state["mat"], state["go"], state["ge"])
        return [t["score"], t["ref_end"], t["read_end"], t["status"]]
    if kind == "sw_host":
        t = state["t"]
        return list(native.sw_batch_host(t["q"], t["qoff"], t["qlen"], t["s"], t["soff"],
                                         t["slen"], state["mat"], state["go"], state["ge"]))
    if kind == "extend":
        return list(state["ix"].sa_hsp(state["queries"], state["query"], state["at"],
                                       state["row"], state["mat"]))
    out = state["ix"].search(state["queries"], state["mat"], **state["opts"])
    return {**{name: out[name] for name in _PER_QUERY}, **_hit_tables(out, state["width"])}


def _mean(median, lo, hi):
    """Mean of the clipped log-normal lengths."""
    z = (np.arange(2000) + 0.5) / 2000
    x = np.exp(math.log(median) + SIGMA * np.sqrt(2) * torch.erfinv(
        torch.from_numpy(2 * z - 1)).numpy())
    return float(np.clip(x, lo, hi).mean())


def work(case):
    """Cells of the alignments at 10 integer operations each (the additions
    and maxima of the three affine recurrences); inputs read and results
    written once."""
    kind = case["kind"]
    if kind in ("sw_device", "sw_host"):
        q = _mean(case["q_median"], case["q_lo"], case["q_hi"])
        s = _mean(case["s_median"], case["s_lo"], case["s_hi"])
        return {"bytes": case["pairs"] * (q + s + 40), "flops": 10 * case["pairs"] * q * s}
    p = _mean(300, 50, 2000)
    if kind == "index":
        n = case["proteins"] * (p + 1)
        return {"bytes": 9 * n, "flops": 0}
    if kind == "extend":
        return {"bytes": case["triples"] * (16 + 8 + 8 + 64), "flops": case["triples"] * 64}
    # one SA row, one text sector and one cursor per popped row: 7 pops per
    # query residue in 50,000 proteins and 13 in 150,000; 0.13 and 0.4
    # alignments (BLOSUM62; more under softer matrices)
    residues = _mean(case["q_median"], case["q_lo"], case["q_hi"]) * case["queries"]
    share = case["proteins"] / 150_000
    pops, pairs = 13 * math.sqrt(share) * residues, 0.4 * share * residues
    cells = pairs * p * residues / case["queries"]
    return {"bytes": 72 * pops + pairs * p + 2 * residues, "flops": 10 * cells}


def tolerance(case):
    return "exact"


# ---------------------------------------------------------- 64-bit references


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sw_device", "sw_host"):
        if case["pairs"] * case["q_hi"] * case["s_hi"] > 1.2e11:
            return None
        return _align(_pairs(case, seed), native.matrix(case["matrix"]), case["gap_open"],
                      case["gap_extend"])
    if kind == "index" and case["proteins"] <= 40_000:
        return _suffixes(_database(case["proteins"], seed)[3].T)
    return None


def _align(t, mat, go, ge):
    """Affine local alignment, column by column over all pairs at once."""
    n, rows, cols = len(t["qlen"]), int(t["qlen"].max()), int(t["slen"].max())
    r = torch.arange(rows, device=DEV)
    pos = t["qoff"][:, None] + r.clamp(max=rows)
    q = t["q"][pos.clamp(max=len(t["q"]) - 1)].long()
    pad = r[None, :] >= t["qlen"][:, None]
    m = torch.from_numpy(mat.astype(np.int64)).to(DEV).reshape(-1)
    H = torch.zeros(n, rows, dtype=torch.int64, device=DEV)
    E = torch.zeros_like(H)
    best = torch.zeros(n, dtype=torch.int64, device=DEV)
    end, read = torch.full_like(best, -1), torch.zeros_like(best)
    for c in range(cols):
        on = c < t["slen"]
        s = t["s"][(t["soff"] + c).clamp(max=len(t["s"]) - 1)].long()
        D = torch.nn.functional.pad(H[:, :-1], (1, 0)) + m[s[:, None] * 25 + q]
        X = torch.maximum(D.masked_fill_(pad, -1000), E).clamp_(min=0)
        F = torch.cummax(X + ge * r, 1).values[:, :-1] - (go + ge * r[:-1])
        H = torch.maximum(X, torch.nn.functional.pad(F, (1, 0)))
        E = torch.maximum(E - ge, H - go)
        top, row = H.masked_fill(pad, 0).max(1)
        row = torch.argmax((H == top[:, None]).to(torch.int8), 1)
        rise = on & (top > best)
        best = torch.where(rise, top, best)
        end = torch.where(rise, c, end)
        read = torch.where(rise, row, read)
    drop = best >= 32767
    if bool(drop.any()):
        best, end, read = best.clamp(max=32767), end.masked_fill(drop, -1), read.masked_fill(drop, -1)
    return [best, end, read, drop.long()]


def _suffixes(T):
    """Suffix array by prefix doubling."""
    n = len(T)
    rank = torch.from_numpy(T.astype(np.int64)).to(DEV)
    h = 1
    while True:
        key = rank * (n + 256) + torch.nn.functional.pad(rank[h:] + 1, (0, min(h, n)))[:n]
        key, sa = torch.sort(key)
        new = torch.nn.functional.pad(torch.cumsum((key[1:] != key[:-1]).long(), 0), (1, 0))
        rank = torch.empty_like(new).scatter_(0, sa, new)
        if int(new[-1]) == n - 1:
            return sa
        h *= 2
