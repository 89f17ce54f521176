"""The band kernel at the edges of its passes, windows and blocks, against the oracle: the winner's
ends of a scan over one pair of sequences, and lone long pairs on one block, several, and two rounds
of 8-row passes (src/database.rs:186-197, src/kernel.rs:331-397)."""
import numpy as np
import pytest

import hyalite_b200 as hy
import pyoracle as o
from conftest import ALL_MODES
from gpu_helpers import BLOSUM62

pytestmark = pytest.mark.gpu

DNA = [2 if a == b else -1 for a in range(4) for b in range(4)]


@pytest.mark.parametrize("mode", ALL_MODES)
@pytest.mark.parametrize("al,mat", [(4, DNA), (20, BLOSUM62)])
def test_winner_ends_at_pass_and_window_edges(mode, al, mat):
    """128-row passes, 16-pair windows, 32-lane skew: widths around multiples of 32 columns and their
    odd neighbours, query lengths around multiples of 128, pairs of unequal halves, planted copies."""
    rng = np.random.default_rng(17 * mode + al)
    for m in (1, 4, 127, 128, 129, 257, 513, 641, 1100):
        q = rng.integers(0, al, m)
        for w0, w1 in ((1, 1), (2, 1), (31, 30), (32, 33), (34, 3), (63, 65), (97, 64), (129, 200), (321, 5)):
            a, b = rng.integers(0, al, w0), rng.integers(0, al, w1)
            k = min(w0, m, 40)
            a[w0 - k:] = q[m - k:]
            seqs = [list(a), list(b)]
            db = (hy.Database.builder().sequences(seqs).scoring(hy.Scoring(al, mat, 11, 1)).mode(hy.Mode(mode))
                  .search_type(hy.SearchType.ScoreEnd).max_query_len(1100).build())
            h = db.scan(hy.Scratch(db), q)
            want = o.OracleDb(seqs, mat, al, 11, 1, mode, 1).scan(list(q))
            assert (h.score, h.db_index, h.query_end, h.target_end) == want, (m, w0, w1)


@pytest.mark.parametrize("mode", ALL_MODES)
def test_lone_pair_at_block_edges(mode):
    """4 passes of 128 rows a block up to 8 blocks (512 and 4096 rows and one more), more warps a block
    beyond, and 8-row passes past 16 warps a block; unrelated and repeated targets (ties)."""
    rng = np.random.default_rng(400 + mode)
    sc = hy.Scoring(20, BLOSUM62, 11, 1)
    for m, n in ((512, 2049), (513, 2047), (640, 1700), (1025, 1030), (4096, 270), (4097, 259), (9000, 131), (16500, 65)):
        q = rng.integers(0, 20, m)
        t = rng.integers(0, 20, n)
        k = min(m, n // 3)
        t[:k] = t[n - k:] = q[:k]
        h = hy.align_pair(q, t, sc, hy.Mode(mode), hy.SearchType.ScoreEnd)
        assert (h.score, h.query_end, h.target_end) == o.align_pair(list(q), list(t), BLOSUM62, 20, 11, 1, mode), (m, n)
