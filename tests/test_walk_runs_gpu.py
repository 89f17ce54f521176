"""The traceback walk, which takes a run of up to 32 operations at a time, at the lengths where a run
fills the warp or ends beside it, against the oracle (src/align.rs:345-420)."""
import numpy as np
import pytest

import pyoracle as o
from conftest import ALL_MODES, identity_matrix

import hyalite_b200 as hy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ALL_MODES)
@pytest.mark.parametrize("ge", [0, 1])
def test_runs_at_warp_edges(mode, ge):
    """Matches, insertions and deletions in runs of 1 to 97, each kind of gap in front, inside and behind,
    and in local mode an end inside a run."""
    rng = np.random.default_rng(10 * mode + ge)
    mat = identity_matrix(4, 5, -4)
    sc = hy.Scoring(4, mat, 3, ge)
    for run in (1, 2, 31, 32, 33, 63, 64, 65, 97):
        for gap in (1, 31, 32, 33, 64, 97):
            parts = [list(rng.integers(0, 4, n)) for n in (run, 40, run)]
            junk = list(rng.integers(0, 4, gap))
            whole = parts[0] + parts[1] + parts[2]
            gapped = parts[0] + junk + parts[1] + parts[2]
            for q, t in ((whole, gapped), (gapped, whole), (whole, junk + gapped), (junk + whole + junk, gapped),
                         (whole, whole[run // 2:] + junk)):
                got = hy.align(q, t, sc, hy.Mode(mode), hy.USIZE_MAX).as_tuple()
                assert got == o.traceback(q, t, mat, 4, 3, ge, mode), (run, gap, len(q), len(t))


@pytest.mark.parametrize("mode", ALL_MODES)
@pytest.mark.parametrize("m", [129, 257, 600])
def test_longest_targets_beside_the_fill(mode, m):
    """Databases whose longest targets run as stripes beside the fill of the rest: 20 and 60 targets, one to
    many of them long, an empty one, ties, against the oracle."""
    rng = np.random.default_rng(1000 * mode + m)
    mat = identity_matrix(4, 2, -1)
    q = list(rng.integers(0, 4, m))
    for n_long, n_short in ((1, 19), (7, 53), (20, 0)):
        seqs = [list(rng.integers(0, 4, int(n))) for n in rng.integers(1, 60, n_short)]
        seqs += [list(rng.integers(0, 4, int(n))) + q[m // 3:] for n in rng.integers(900, 2500, n_long)]
        seqs += [[], list(seqs[-1])]
        seqs = [seqs[i] for i in rng.permutation(len(seqs))]
        db = (hy.Database.builder().sequences(seqs).scoring(hy.Scoring(4, mat, 2, 1)).mode(hy.Mode(mode))
              .search_type(hy.SearchType.alignment(hy.USIZE_MAX)).max_query_len(m).build())
        sc = hy.Scratch(db)
        for _ in range(2):
            out = []
            db.scan_all_aligned(sc, q, out)
            assert len(out) == len(seqs)
            for a, t in zip(out, seqs):
                assert a.as_tuple() == o.traceback(q, t, mat, 4, 2, 1, mode), (n_long, len(t))
