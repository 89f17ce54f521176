"""hy_scratch_profile: every main kernel of a scan is timed and its cells counted, whatever forms its items take
(the bulk kernel, a warp each, the band kernel; int32 items either way), so the classes' cells together are the
scan's."""
import ctypes as C

import numpy as np
import pytest

import hyalite_b200 as hy
from gpu_helpers import BLOSUM62
from hyalite_b200 import _abi

pytestmark = pytest.mark.gpu


def _profile(db, sc, call):
    _abi.lib.hy_scratch_profile(sc._h, 1)
    call()
    ms, n, cells, every = (C.c_double * 3)(), (C.c_uint64 * 3)(), (C.c_double * 3)(), C.c_uint64()
    assert _abi.lib.hy_scratch_profile_read(sc._h, ms, n, cells, C.byref(every)) == 0
    _abi.lib.hy_scratch_profile(sc._h, 0)
    return list(ms), list(n), list(cells), every.value


# A few long targets (bands alone), log-normal ones (bands, a warp each, the bulk), many equal ones (the bulk),
# and the same with scores that need int32.
CASES = [("long", 1), ("mixed", 1), ("equal", 1), ("long", 600), ("equal", 600), ("mixed", 40)]


@pytest.mark.parametrize("kind,scale", CASES)
@pytest.mark.parametrize("ends", [False, True])
def test_all_items_are_timed(kind, scale, ends):
    rng = np.random.default_rng(len(kind))
    lens = {"long": rng.integers(900, 2000, 24), "equal": np.full(20_000, 150),
            "mixed": np.clip(np.exp(np.log(150) + 0.9 * rng.standard_normal(12_000)), 5, 4000).astype(int)}[kind]
    off = np.zeros(len(lens) + 1, np.uint64)
    off[1:] = np.cumsum(lens)
    res = rng.integers(0, 20, int(off[-1])).astype(np.uint8)
    sc_ = hy.Scoring(20, [int(v) * scale for v in BLOSUM62], 11 * scale, scale)
    m = 400
    db = (hy.Database.builder().sequences_concat(res, off).scoring(sc_).mode(hy.Mode.Sw)
          .search_type(hy.SearchType.ScoreEnd).max_query_len(m).build())
    sc, q = hy.Scratch(db), rng.integers(0, 20, m).astype(np.uint8)
    ms, n, cells, every = _profile(db, sc, lambda: db.scan_all_array(sc, q) if ends else db.scan(sc, q))
    f = (C.c_uint32 * 5)()
    _abi.lib.hy_debug_scan_forms(db._h, m, int(ends), f)
    want = [int(f[4] > 0), int(f[0] > 0), int(f[2] > 0) + int(f[3] > 0)]
    assert n == want and sum(want) > 0, (n, list(f))
    assert sum(cells) == float(m) * float(off[-1]) or f[0] > 0
    assert sum(cells) >= float(m) * float(off[-1])  # (a pair cut by the int32 split counts its shorter half twice)
    for t, k in zip(ms, n):
        assert (t > 0.0) == (k > 0)
    assert every >= 2 * sum(n)
