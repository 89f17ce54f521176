"""The forms a scan splits its items over (the band kernel, a warp a pair, the bulk kernel; int32 items
either way) against the oracle, on databases whose length mix puts pairs in each."""
import ctypes as C

import numpy as np
import pytest

import hyalite_b200 as hy
import pyoracle as o
from conftest import ALL_MODES
from gpu_helpers import BLOSUM62
from hyalite_b200 import _abi

pytestmark = pytest.mark.gpu

DNA = [2 if a == b else -1 for a in range(4) for b in range(4)]


def _forms(db, qlen, ends):
    out = (C.c_uint32 * 5)()
    _abi.lib.hy_debug_scan_forms(db._h, qlen, int(ends), out)
    return tuple(out)


@pytest.mark.parametrize("mode", ALL_MODES)
@pytest.mark.parametrize("al,mat", [(4, DNA), (20, BLOSUM62)])
def test_every_form_matches_the_oracle(al, mat, mode):
    """Best hit, every score and every target's ends for query lengths that take each wide shape (64,
    128, 256, 384, 512 rows, several passes of 256 and of 512) and their neighbours."""
    rng = np.random.default_rng(31 * al + mode)
    queries = [rng.integers(0, al, m) for m in (64, 65, 129, 384, 500, 700, 1030)]
    lens = np.clip(np.exp(np.log(60) + 0.8 * rng.standard_normal(12_000)), 5, 2500).astype(int)
    seqs = [rng.integers(0, al, n) for n in lens]
    for k, q in enumerate(queries):  # planted pieces, some twice: ties by index and by column
        for i in (3 * k, 3 * k + 1):
            n = min(len(q), len(seqs[i]) // 2)
            seqs[i][:n] = seqs[i][len(seqs[i]) - n:] = q[:n]
    seqs = [list(s) for s in seqs]
    db = (hy.Database.builder().sequences(seqs).scoring(hy.Scoring(al, mat, 11, 1)).mode(hy.Mode(mode))
          .search_type(hy.SearchType.ScoreEnd).max_query_len(1030).build())
    ref = o.OracleDb(seqs, mat, al, 11, 1, mode, 1)
    sc = hy.Scratch(db)
    used = np.zeros(5, np.int64)
    for q in queries:
        want = ref.scan_all(list(q))
        hits = db.scan_all_array(sc, q)
        got = [(h.score, h.db_index, None if h.query_end < 0 else h.query_end, None if h.target_end < 0 else h.target_end)
               for h in hits]
        assert got == [tuple(w) for w in want], [(len(q), g, w) for g, w in zip(got, want) if g != tuple(w)][:3]
        assert list(db.scan_scores_array(sc, q)) == [w[0] for w in want], len(q)
        h = db.scan(sc, q)
        best = max(want, key=lambda w: (w[0], -w[1]))
        assert (h.score, h.db_index, h.query_end, h.target_end) == tuple(best), len(q)
        used += np.minimum(_forms(db, len(q), False), 1) + np.minimum(_forms(db, len(q), True), 1)
    assert np.all(used[2:] > 0), used  # the band kernel, a warp a pair and the bulk kernel all ran
