"""The warp form of the --blasttab statistics where it has edges: bands wider
than the 32 rows of a step block and wider than the subject, segments around
32 rows, bands that double, and inputs no forward pass gives (another score,
gap costs the batch alignment does not take), against the host restatement."""
import ctypes

import numpy as np
import pytest

from test_stats_gpu import FIELDS, St, _device_stats, _same_double
from topaz_b200 import native, synth

pytestmark = pytest.mark.gpu


def _check(torch, ps, mat, go, ge, fwd):
    got = _device_stats(torch, ps, mat, go, ge, fwd)
    L = native.lib()
    L.tpzh_align_stats.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_int32,
                                   ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int32,
                                   ctypes.c_int32, ctypes.c_int32, ctypes.POINTER(St)]
    m = np.ascontiguousarray(mat, np.int8)
    for i in range(ps.n):
        q = np.ascontiguousarray(ps.q[ps.qoff[i]:ps.qoff[i] + ps.qlen[i]])
        s = np.ascontiguousarray(ps.s[ps.soff[i]:ps.soff[i] + ps.slen[i]])
        h = St()
        L.tpzh_align_stats(q.ctypes.data, len(q), s.ctypes.data, len(s), m.ctypes.data, go, ge,
                           int(fwd[2][i]), int(fwd[1][i]), int(fwd[0][i]), ctypes.byref(h))
        assert tuple(int(got[k][i]) for k in FIELDS) == tuple(getattr(h, k) for k in FIELDS), i
        assert _same_double(got["identity"][i], h.identity), i


def _gapped_pairs():
    """Subjects that are the query with a piece cut out or put in, at sizes
    around the row blocks."""
    rng = np.random.default_rng(5)
    qs, ss = [], []
    for n in (31, 32, 33, 63, 64, 65, 97, 300, 900):
        for gap in (0, 1, 2, 5, 31, 33, 120):
            q = rng.integers(0, 20, n).astype(np.int8)
            at = n // 2
            ins = rng.integers(0, 20, gap).astype(np.int8)
            s = np.concatenate([q[:at], ins, q[at:]])
            noise = rng.random(len(s)) < 0.15
            s[noise] = rng.integers(0, 20, int(noise.sum()))
            qs += [q, s]
            ss += [s, q]
    ql = np.array([len(x) for x in qs], np.int32)
    sl = np.array([len(x) for x in ss], np.int32)
    return synth.PairSet(np.concatenate(qs), (np.cumsum(ql) - ql).astype(np.int64), ql, np.concatenate(ss),
                         (np.cumsum(sl) - sl).astype(np.int64), sl, 0)


@pytest.mark.parametrize("go,ge", [(11, 1), (2, 1), (1, 0), (30, 0)])
def test_bands_around_the_row_blocks(cuda, go, ge):
    ps, mat = _gapped_pairs(), synth.matrix("BLOSUM62")
    sc, re_, rd, st = native.sw_batch_host(ps.q, ps.qoff, ps.qlen, ps.s, ps.soff, ps.slen, mat, go, ge)
    assert (st == native.TPZ_SW_OK).all()
    _check(cuda, ps, mat, go, ge, (sc, re_, rd))


def test_launch_count_stays_the_batch_calls(cuda):
    ps, mat = _gapped_pairs(), synth.matrix("BLOSUM62")
    t = {k: cuda.from_numpy(np.ascontiguousarray(getattr(ps, k))).cuda() for k in ("q", "s")}
    for k in ("qoff", "qlen", "soff", "slen"):
        t[k] = cuda.from_numpy(np.tile(getattr(ps, k), 50)).cuda()
    for k in ("score", "ref_end", "read_end", "status"):
        t[k] = cuda.empty(50 * ps.n, dtype=cuda.int32, device="cuda")
    native.sw_batch_torch(t, mat)                    # another form than the statistics' batch
    counted = native.last_launches()
    sc, re_, rd = (t[k][:ps.n].cpu().numpy() for k in ("score", "ref_end", "read_end"))
    _device_stats(cuda, ps, mat, 11, 1, (sc, re_, rd))
    assert native.last_launches() == counted > 6


@pytest.mark.parametrize("shift,go,ge", [(-1, 11, 1), (0, 2, 2), (0, 1, 3)])
def test_inputs_no_forward_pass_gives(cuda, shift, go, ge):
    ps, mat = _gapped_pairs(), synth.matrix("BLOSUM62")
    sc, re_, rd, _ = native.sw_batch_host(ps.q, ps.qoff, ps.qlen, ps.s, ps.soff, ps.slen, mat, 11, 1)
    _check(cuda, ps, mat, go, ge, (np.maximum(sc + shift, 1), re_, rd))


@pytest.mark.parametrize("go,ge", [(11, 1), (2, 2)])
def test_bytes_outside_the_alphabet(cuda, go, ge):
    # they score -64, as in the forward pass: the same columns as for a letter
    # whose scores are all -64
    ps, mat = _gapped_pairs(), synth.matrix("BLOSUM62").copy()
    mat[24, :] = mat[:, 24] = -64
    rng = np.random.default_rng(9)
    known = synth.PairSet(ps.q.copy(), ps.qoff, ps.qlen, ps.s.copy(), ps.soff, ps.slen, 0)
    for i in range(ps.n):                            # in half of the pairs each
        buf, off, n = (ps.q, ps.qoff, ps.qlen) if i % 4 < 2 else (ps.s, ps.soff, ps.slen)
        at = off[i] + rng.integers(0, n[i], 1 + n[i] // 40)
        buf[at] = rng.choice(np.array([25, 30, 127, -1, -128], np.int8), len(at))
        (known.q if i % 4 < 2 else known.s)[at] = 24
    fwd = native.sw_batch_host(ps.q, ps.qoff, ps.qlen, ps.s, ps.soff, ps.slen, mat, 11, 1)
    same = native.sw_batch_host(known.q, known.qoff, known.qlen, known.s, known.soff, known.slen, mat, 11, 1)
    assert all((x == y).all() for x, y in zip(fwd, same)) and (fwd[3] == 0).all()
    got = _device_stats(cuda, ps, mat, go, ge, fwd[:3])
    want = _device_stats(cuda, known, mat, go, ge, fwd[:3])
    for k in FIELDS:
        assert (got[k] == want[k]).all(), k
    assert got["identity"].tobytes() == want["identity"].tobytes()
    assert (got["length"] > 0).sum() > ps.n // 2 or go == ge
