"""Scans whose bands would leave a scheduler few warps (large alphabets: a band's slices fill an SM's shared
memory): the estimate that splits a scan's items keeps them out of the band kernel, and puts the same shapes of
a small alphabet there; results against the oracle."""
import ctypes as C

import numpy as np
import pytest

import hyalite_b200 as hy
import pyoracle as o
from hyalite_b200 import _abi

pytestmark = pytest.mark.gpu


def _scan(al, scale, lens, m, mode):
    rng = np.random.default_rng(al + m)
    mat = rng.integers(-4, 4, (al, al))
    mat = np.triu(mat) + np.triu(mat, 1).T
    mat[np.diag_indices(al)] = 7
    mat = [int(v) * scale for v in mat.reshape(-1)]
    q = rng.integers(0, al, m)
    seqs = [list(rng.integers(0, al, int(n))) for n in lens]
    db = (hy.Database.builder().sequences(seqs).scoring(hy.Scoring(al, mat, 11 * scale, scale)).mode(mode)
          .search_type(hy.SearchType.ScoreEnd).max_query_len(m).build())
    got = [h.score for h in db.scan_all_array(hy.Scratch(db), q)]
    assert got == [w[0] for w in o.OracleDb(seqs, mat, al, 11 * scale, scale, int(mode), 1).scan_all(list(q))]
    out = (C.c_uint32 * 5)()
    _abi.lib.hy_debug_scan_forms(db._h, m, 0, out)
    return tuple(out)


@pytest.mark.parametrize("al,band", [(20, 1), (250, 0)])
def test_72_int32_items(al, band):
    assert _scan(al, 400, np.full(72, 150), 777, hy.Mode.Sw)[:2] == (72, band)


def test_many_int32_items_on_clusters():
    """50 letters, 12 passes on three blocks, two blocks an SM."""
    lens = np.sort(np.exp(np.log(300) + 0.8 * np.random.default_rng(1).standard_normal(1300)).clip(40, 4000).astype(int))
    f = _scan(50, 400, lens, 1439, hy.Mode.Shw)
    assert f[0] > 1000 and f[1] == 0, f


@pytest.mark.parametrize("al", [4, 150])
def test_pairs_of_one_block_bands(al):
    """39 residues: one warp a block, at 150 letters one block an SM."""
    f = _scan(al, 1, np.random.default_rng(2).integers(50, 301, 1627), 39, hy.Mode.Sw)
    assert f[0] == 0 and (f[2] == 0 or al == 4), f
