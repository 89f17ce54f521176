"""align_pairs' wide form (a warp an item) at the edges of its passes, beside the narrow form and the long
pairs' stripes, against the oracle (src/kernel.rs:429-452)."""
import numpy as np
import pytest

import pyoracle as o
from conftest import ALL_MODES, DNA
from gpu_helpers import BLOSUM62

import hyalite_b200 as hy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ALL_MODES)
@pytest.mark.parametrize("al,mat", [(4, DNA), (20, BLOSUM62)])
def test_wide_items_at_pass_edges(mode, al, mat):
    """Queries of 1 to 1030 residues around the passes of 128 and 256 rows, targets of 0 to 900, odd and even
    counts of a length; then the same pairs behind 3,000 short ones, and with two long pairs."""
    rng = np.random.default_rng(7 * mode + al)
    qs, ts = [], []
    for m in (0, 1, 4, 5, 127, 128, 129, 255, 256, 257, 300, 511, 512, 513, 1030):
        for n in (0, 1, 31, 32, 33, 150, 900)[: 6 + (m % 2)]:
            q = rng.integers(0, al, m)
            t = rng.integers(0, al, n)
            k = min(m, n // 2)
            t[:k] = t[n - k:] = q[:k]  # a repeated piece: ties by column
            qs.append(list(q))
            ts.append(list(t))
    short_q = [list(rng.integers(0, al, int(n))) for n in rng.integers(1, 80, 3000)]
    short_t = [list(rng.integers(0, al, int(n))) for n in rng.integers(1, 90, 3000)]
    long_q = [list(rng.integers(0, al, n)) for n in (1100, 700)]
    long_t = [list(rng.integers(0, al, n)) for n in (1000, 1600)]
    for a, b in ((qs, ts), (short_q + qs, short_t + ts), (long_q + qs, long_t + ts)):
        for st in (0, 1):
            out = []
            hy.align_pairs(list(zip(a, b)), hy.Scoring(al, mat, 11, 1), hy.Mode(mode), hy.SearchType(st), out)
            status, want, _ = o.align_pairs(a, b, mat, al, 11, 1, mode, st)
            assert status == 0
            got = [(h.score, h.db_index, h.query_end, h.target_end) for h in out]
            assert got == want, [(i, len(a[i]), len(b[i]), got[i], want[i]) for i in range(len(a)) if got[i] != want[i]][:4]
