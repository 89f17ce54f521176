"""int32 items of a scan in each of their forms (the band kernel, a warp each with two columns a step, a warp
each with one), and pairs a warp each in several passes of 512 rows, against the oracle in every mode."""
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


def _matrix(al, scale):
    rng = np.random.default_rng(al)
    m = rng.integers(-4, 4, (al, al))
    m = np.triu(m) + np.triu(m, 1).T
    m[np.diag_indices(al)] = rng.integers(4, 12, al)
    return [int(v) * scale for v in m.reshape(-1)]


def _forms(db, qlen, ends):
    out = (C.c_uint32 * 5)()
    _abi.lib.hy_debug_scan_forms(db._h, qlen, int(ends), out)
    return tuple(out)


def _build(seqs, mat, al, go, ge, mode, mql):
    return (hy.Database.builder().sequences(seqs).scoring(hy.Scoring(al, mat, go, ge)).mode(hy.Mode(mode))
            .search_type(hy.SearchType.ScoreEnd).max_query_len(mql).build())


def _check(db, seqs, mat, al, go, ge, mode, q):
    want = o.OracleDb(seqs, mat, al, go, ge, mode, 1).scan_all(list(q))
    sc = hy.Scratch(db)
    got = [(h.score, h.db_index, None if h.query_end < 0 else h.query_end, None if h.target_end < 0 else h.target_end)
           for h in db.scan_all_array(sc, q)]
    assert got == [tuple(w) for w in want], [(g, w) for g, w in zip(got, want) if g != tuple(w)][:3]
    assert list(db.scan_scores_array(sc, q)) == [w[0] for w in want]
    h = db.scan(sc, q)
    best = max(want, key=lambda w: (w[0], -w[1]))
    assert (h.score, h.db_index, h.query_end, h.target_end) == tuple(best)


def _planted(rng, al, lens, q):
    """Sequences of these lengths, every fifth with a piece of the query at both ends (ties by column)."""
    seqs = [rng.integers(0, al, int(n)) for n in lens]
    for s in seqs[::5]:
        n = min(len(q), len(s) // 2)
        s[:n] = s[len(s) - n:] = q[:n]
    seqs[1] = seqs[0].copy()  # a tie by index
    return [list(s) for s in seqs]


# (targets, lengths from, to, query, whether the int32 items take the band kernel)
SHAPES = [(30, 900, 2200, 700, 1), (4000, 90, 110, 300, 0), (3000, 150, 260, 520, 0), (1500, 380, 420, 520, 0),
          (4000, 1, 60, 600, 0)]


@pytest.mark.parametrize("mode", ALL_MODES)
@pytest.mark.parametrize("n,lo,hi,m,band", SHAPES)
def test_int32_items(mode, n, lo, hi, m, band):
    """Few long items (the band kernel), many of about 100, 200 and 400 columns, and many very short ones in
    two passes; the scoring is scaled so that all or most need int32."""
    rng = np.random.default_rng(n + m + mode)
    scale = 600
    mat = _matrix(20, scale)
    q = rng.integers(0, 20, m)
    seqs = _planted(rng, 20, rng.integers(lo, hi, n), q)
    db = _build(seqs, mat, 20, 11 * scale, scale, mode, m)
    for ends in (False, True):
        f = _forms(db, m, ends)
        assert f[0] > n // 2 and f[1] == band, f
    _check(db, seqs, mat, 20, 11 * scale, scale, mode, q)


@pytest.mark.parametrize("mode", ALL_MODES)
@pytest.mark.parametrize("m", [400, 513])
def test_int32_items_of_a_large_alphabet(mode, m):
    """50 letters: a band block holds few warps, so many items keep a warp each, and in local mode the copies
    of the two-column sweep do not fit beside the pass slices."""
    rng = np.random.default_rng(m + mode)
    scale = 600
    mat = _matrix(50, scale)
    q = rng.integers(0, 50, m)
    seqs = _planted(rng, 50, rng.integers(100, 600, 1200), q)
    db = _build(seqs, mat, 50, 11 * scale, scale, mode, m)
    f = _forms(db, m, True)
    assert f[0] > 1000 and f[1] == 0, f
    _check(db, seqs, mat, 50, 11 * scale, scale, mode, q)


@pytest.mark.parametrize("mode", ALL_MODES)
@pytest.mark.parametrize("al,mat", [(4, DNA), (20, BLOSUM62)])
def test_pairs_a_warp_each_in_several_passes_of_512_rows(mode, al, mat):
    """Queries of 1000 to 1536 residues: two and three passes of 512 rows (blocks of 512 threads for 20
    letters), 256-row passes in local mode with ends there."""
    rng = np.random.default_rng(11 * mode + al)
    lens = rng.integers(30, 90, 1200)
    for m in (1000, 1024, 1500, 1536):
        q = rng.integers(0, al, m)
        seqs = _planted(rng, al, lens, q)
        db = _build(seqs, mat, al, 11, 1, mode, m)
        for ends in (False, True):
            f = _forms(db, m, ends)
            assert f[0] == 0 and f[3] > 0, (m, f)
        _check(db, seqs, mat, al, 11, 1, mode, q)
