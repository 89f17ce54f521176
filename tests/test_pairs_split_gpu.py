"""Which of a call's items take align_pairs' wide form (a warp an item): none of many reads, most of a few
ragged proteins, none of the column-maxima form, counted over the call's chunks; results against the oracle
(src/kernel.rs:429-452)."""
import numpy as np
import pytest

import hyalite_b200 as hy
import pyoracle as o
from conftest import DNA
from gpu_helpers import BLOSUM62
from hyalite_b200 import _abi

pytestmark = pytest.mark.gpu


def _off(lens):
    off = np.zeros(len(lens) + 1, np.uint64)
    off[1:] = np.cumsum(lens)
    return off


def _run(al, mat, ql, tl, check):
    rng = np.random.default_rng(len(ql) + al)
    qo, to = _off(ql), _off(tl)
    q, t = rng.integers(0, al, int(qo[-1])).astype(np.uint8), rng.integers(0, al, int(to[-1])).astype(np.uint8)
    hits, (err, _) = hy.align_pairs_arrays(q, qo, t, to, hy.Scoring(al, mat, 11, 1), hy.Mode.Hw, hy.SearchType.ScoreEnd)
    assert err is None
    wide = _abi.lib.hy_debug_pairs_wide_items()
    for k in check:
        want = o.align_pair(list(q[qo[k]:qo[k + 1]]), list(t[to[k]:to[k + 1]]), mat, al, 11, 1, int(hy.Mode.Hw))
        assert (hits[k].score, hits[k].query_end, hits[k].target_end) == want, k
    return wide


def test_many_reads_keep_the_narrow_form():
    n = 60_000  # three chunks
    tl = np.random.default_rng(1).integers(200, 501, n)
    assert _run(4, DNA, np.full(n, 150), tl, range(0, n, 1999)) == 0


@pytest.mark.parametrize("n", [37, 2000, 40_000])
def test_ragged_proteins_take_the_wide_form(n):
    """One pair of every ten long; 40,000 pairs are two chunks, whose sums run on the host threads."""
    rng = np.random.default_rng(n)
    ql, tl = (np.where(rng.random(n) < 0.1, rng.integers(400, 900, n), rng.integers(20, 60, n)) for _ in range(2))
    assert _run(20, BLOSUM62, ql, tl, range(0, n, max(1, n // 40))) > 0


def test_column_maxima_keep_the_narrow_form():
    rng = np.random.default_rng(3)
    ql, tl = rng.integers(20, 600, 50), rng.integers(20, 900, 50)
    qo, to = _off(ql), _off(tl)
    q, t = rng.integers(0, 4, int(qo[-1])).astype(np.uint8), rng.integers(0, 4, int(to[-1])).astype(np.uint8)
    hy.align_pairs_position_max_arrays(q, qo, t, to, hy.Scoring(4, DNA, 11, 1), 20, np.empty(int(to[-1]), np.int32))
    assert _abi.lib.hy_debug_pairs_wide_items() == 0
