"""The recurrence of the batch kernels against the lane-length oracle.

The kernels run one pass without SSW's in-lane vertical-gap term, because H
does not depend on it (csrc/sw_core.cuh).  Here that is checked on the CPU
where it could fail if it were false: few letters, matrices of any sign,
gap costs down to (1, 0), so that vertical gaps next to horizontal ones and
ties are common."""
import numpy as np
import pytest

import oracle


def _one_pass(q, s, mat, go, ge):
    """(score, ref_end, read_end) with E and F fed by X alone; rows of E that
    equal m - go after a column that raises the maximum to m give read_end."""
    rows = len(q)
    H, E = np.zeros(rows + 1, np.int64), np.full(rows, -go, np.int64)
    best, end, read = 0, -1, 0
    for c, letter in enumerate(s):
        X = np.maximum(H[:-1] + mat[letter, q], E)
        F = np.empty(rows, np.int64)
        f = 0
        for r in range(rows):
            F[r] = f
            f = max(f - ge, X[r] - go)
        E = np.maximum(E - ge, X - go)
        H[1:] = np.maximum(np.maximum(X, F), 0)
        if X.max() > best:
            best, end = int(X.max()), c
            read = int(np.flatnonzero(E == best - go)[0])
    return best, end, read


@pytest.mark.parametrize("letters,top", [(1, 3), (2, 3), (2, 12), (3, 6), (4, 40), (20, 11)])
def test_one_pass_equals_the_lane_passes(letters, top):
    rng = np.random.default_rng(letters * 100 + top)
    for _ in range(60):
        q = rng.integers(0, letters, int(rng.integers(1, 90))).astype(np.int8)
        s = rng.integers(0, letters, int(rng.integers(0, 90))).astype(np.int8)
        mat = rng.integers(-8, top + 1, (25, 25)).astype(np.int8)
        ge = int(rng.integers(0, 4))
        go = ge + 1 + int(rng.integers(0, 4))
        text = s if len(s) else np.zeros(1, np.int8)
        want = oracle.oracle_sw(q, np.zeros(1, np.int64), np.array([len(q)], np.int32), text,
                                np.zeros(1, np.int64), np.array([len(s)], np.int32), mat, go, ge)
        assert _one_pass(q, s, mat.astype(np.int64), go, ge) == tuple(int(x[0]) for x in want[:3])
