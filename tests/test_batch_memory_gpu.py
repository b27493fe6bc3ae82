"""Device memory of a search batch with stripe boundary rows: sized by the
subjects the batch hits, within a fixed total, and the pairs of a batch whose
subjects are too long for that still give the oracle's results."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from topaz_b200 import alphabet as ab, native, synth

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LONG = 300_000


def _family():
    """60 queries of 1,100 residues that hit 20 proteins of their family,
    an unrelated protein of LONG residues, and one that holds a piece."""
    rng = np.random.Generator(np.random.PCG64(17))
    base = synth.random_residues(rng, 1100)
    family = [synth.mutate(rng, base, 0.7) for _ in range(20)]
    other = synth.random_residues(rng, LONG)
    holds = synth.random_residues(rng, LONG)
    holds[200_000:200_300] = base[400:700]
    queries = [ab.aa_to_internal(np.concatenate([synth.mutate(rng, base, 0.9), synth.random_residues(rng, 60)]))
               for _ in range(60)]
    return family, other, holds, [q.tobytes() for q in queries]


def _index(seqs):
    from topaz_b200 import dbformat
    db = dbformat.build_from_records([(b"p%d" % i, s) for i, s in enumerate(seqs)])
    db.SA = native.sa_build(db.T)
    return db, native.Index(db)


def _child():
    import torch
    family, other, holds, queries = _family()
    used = []
    for extra in (other, holds):
        db, ix = _index(family + [extra])
        mat = native.matrix("BLOSUM62")
        ix.search(queries[:1], mat)                  # context, modules, streams
        free = torch.cuda.mem_get_info()[0]
        r = ix.search(queries, mat)
        assert (np.diff(r["hit_off"]) >= 20).all()
        used.append(free - torch.cuda.mem_get_info()[0])
        del ix
    print(json.dumps(used))


def test_memory_of_a_batch_beside_a_long_protein(cuda):
    # (in a process of its own: the pool keeps what other batches grew it to)
    run = "import sys; sys.path[:0] = %r; import test_batch_memory_gpu as t; t._child()" % [
        ROOT, os.path.join(ROOT, "tests")]
    out = subprocess.run([sys.executable, "-c", run], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    used = json.loads(out.stdout.strip().splitlines()[-1])
    # queries' shares, stored columns, and 60 blocks' boundaries of 1,300 columns
    share = sum(native.query_device_bytes(1160) for _ in range(60)) + native.batch_device_bytes(1024, 0)
    assert used[0] < share + (64 << 20) and used[1] < share + (64 << 20), (used, share)


def test_hits_longer_than_the_boundary_rows(cuda):
    family, _, holds, queries = _family()
    db, ix = _index(family + [holds])
    mat = native.matrix("BLOSUM62")
    r = ix.search(queries, mat)
    longest = [int((r["protein"][a:b] == 20).sum()) for a, b in zip(r["hit_off"], r["hit_off"][1:])]
    assert min(longest) == 1                        # every query hits the long one
    a, b = r["hit_off"][7], r["hit_off"][8]
    ps = db.pstart
    subj = [ab.internal_to_index(db.T[ps[p]:ps[p] + db.ind["protein_len"][p]]) for p in r["protein"][a:b]]
    q = ab.internal_to_index(np.frombuffer(queries[7], np.uint8))
    sl = np.array([len(x) for x in subj], np.int32)
    n = len(subj)
    want = oracle.oracle_sw(q, np.zeros(n, np.int64), np.full(n, len(q), np.int32), np.concatenate(subj),
                            (np.cumsum(sl) - sl).astype(np.int64), sl, mat)
    on = r["gapless_score"][a:b] >= 40
    assert on.sum() >= 16
    for got, w in (("rawscore", 0), ("send", 1), ("qend", 2), ("sw_status", 3)):
        assert (r[got][a:b][on] == want[w][on]).all(), got
