"""Band launches whose shared memory comes within a kilobyte of what a block may have (some alphabets at
some query lengths): the winner's ends of a scan in both pair layouts and int32, and lone long pairs, against
the oracle (src/database.rs:186-197, src/kernel.rs:331-397)."""
import ctypes as C

import numpy as np
import pytest

import hyalite_b200 as hy
import pyoracle as o
from gpu_helpers import hit_tuple
from hyalite_b200 import _abi

pytestmark = pytest.mark.gpu

LIMIT = 227 * 1024


def _matrix(al, scale=1):
    rng = np.random.default_rng(al)
    m = rng.integers(-4, 4, (al, al))
    m = np.triu(m) + np.triu(m, 1).T
    m[np.diag_indices(al)] = 7
    return [int(v) * scale for v in m.reshape(-1)]


def _room(arith, al, qlen):
    out = np.zeros(6, np.uint64)
    assert _abi.lib.hy_debug_band_plan(arith, 0, al, qlen, LIMIT, out.ctypes.data_as(C.POINTER(C.c_uint64))) == 0
    return LIMIT - int(out[5])


@pytest.mark.parametrize("arith,al,qlen", [(0, 28, 6200), (0, 71, 300), (0, 71, 600), (0, 71, 1050), (0, 221, 50),
                                           (1, 11, 300), (1, 11, 600), (2, 30, 11300), (2, 57, 6200), (2, 143, 300),
                                           (2, 218, 150)])
def test_winner_ends(arith, al, qlen):
    assert _room(arith, al, qlen) < 1024
    rng = np.random.default_rng(qlen)
    scale = 3000 if arith == 2 else 1  # every item int32
    mat = _matrix(al, scale)
    q = rng.integers(0, al, qlen)
    seqs = [list(rng.integers(0, al, int(n))) for n in (60, 200, 77, 131)]
    seqs[2][10:50] = q[5:45]
    layout = hy.LayoutChoice.Force(hy.Layout.Precomputed if arith == 1 else hy.Layout.Gathered)
    db = (hy.Database.builder().sequences(seqs).scoring(hy.Scoring(al, mat, 11 * scale, scale)).mode(hy.Mode.Sw)
          .search_type(hy.SearchType.ScoreEnd).layout(layout).max_query_len(qlen).build())
    assert hit_tuple(db.scan(hy.Scratch(db), q)) == o.OracleDb(seqs, mat, al, 11 * scale, scale, 0, 1).scan(list(q))


@pytest.mark.parametrize("al,qlen,near", [(30, 11300, True), (57, 6200, True), (143, 300, True), (9, 19500, False)])
def test_lone_pairs(al, qlen, near):
    """(9 letters: two rounds of 4-row passes, which 8-row passes would take one of.)"""
    assert (_room(2, al, qlen) < 1024) == near
    rng = np.random.default_rng(al)
    q, t = rng.integers(0, al, qlen), rng.integers(0, al, (1 << 20) // qlen + 1)
    h = hy.align_pair(q, t, hy.Scoring(al, _matrix(al), 11, 1), hy.Mode.Sw, hy.SearchType.ScoreEnd)
    assert (h.score, h.query_end, h.target_end) == o.align_pair(list(q), list(t), _matrix(al), al, 11, 1, 0)
