"""The band kernel's blocks giving up on one another's rows: hy_debug_set_row_wait_polls(0) makes every
wait between the blocks of a cluster run out at once (the profile copies still arrive), so a block stops
arming and giving back its ring, the block above it sends the ring blocks it has room for and no more, and
all of them stop at the next cluster barrier. The call reports Timeout, and with the limit restored the
same scratch and the same context give the oracle's results (HY_ERR_TIMEOUT has no counterpart in the
reference, whose scan cannot fail: src/database.rs:79-89)."""
import numpy as np
import pytest

import hyalite_b200 as hy
import pyoracle as o
from conftest import ALL_MODES
from gpu_helpers import BLOSUM62, hit_tuple
from hyalite_b200 import _abi

pytestmark = pytest.mark.gpu


class _RowPolls:
    def __enter__(self):
        _abi.lib.hy_debug_set_row_wait_polls(0)

    def __exit__(self, *exc):
        _abi.lib.hy_debug_set_row_wait_polls(-1)


def _ends(h):
    return (h.score, h.db_index, None if h.query_end < 0 else h.query_end, None if h.target_end < 0 else h.target_end)


def _times_out(call):
    with pytest.raises(hy.Error) as e:
        call()
    assert e.value.kind == "Timeout"


@pytest.mark.parametrize("mode", ALL_MODES)
def test_lone_pair_whose_rows_do_not_arrive(mode):
    """5 passes on two blocks (the shortest such query), 8 blocks, targets of one ring block, of the four a
    ring holds, of one more, and of many."""
    rng = np.random.default_rng(900 + mode)
    sc = hy.Scoring(20, BLOSUM62, 11, 1)
    for m, n in ((520, 2100), (600, 3001), (4096, 260), (4090, 257), (4000, 1500)):
        q, t = rng.integers(0, 20, m), rng.integers(0, 20, n)
        call = lambda: hy.align_pair(q, t, sc, hy.Mode(mode), hy.SearchType.ScoreEnd)  # noqa: E731
        with _RowPolls():
            _times_out(call)
            _times_out(call)
        h = call()
        assert (h.score, h.query_end, h.target_end) == o.align_pair(list(q), list(t), BLOSUM62, 20, 11, 1, mode), (m, n)


@pytest.mark.parametrize("width", [31, 32, 33, 127, 128, 129, 160, 161, 400])
def test_winner_and_band_items_whose_rows_do_not_arrive(width):
    """The winner's ends of a scan (its graph captured under both limits), and a scan whose every item runs on
    the band kernel, at targets around the ring's 16, 64 and 80 column pairs."""
    rng = np.random.default_rng(width)
    seqs = [list(rng.integers(0, 20, width)) for _ in range(3)]
    db = (hy.Database.builder().sequences(seqs).scoring(hy.Scoring(20, BLOSUM62, 11, 1)).mode(hy.Mode.Sw)
          .search_type(hy.SearchType.ScoreEnd).max_query_len(1200).build())
    ref = o.OracleDb(seqs, BLOSUM62, 20, 11, 1, 0, 1)
    sc = hy.Scratch(db)
    q = rng.integers(0, 20, 1200)
    want, want_all = ref.scan(list(q)), ref.scan_all(list(q))
    for _ in range(2):
        assert hit_tuple(db.scan(sc, q)) == want
        assert [_ends(h) for h in db.scan_all_array(sc, q)] == want_all
        with _RowPolls():
            _times_out(lambda: db.scan(sc, q))
    assert hit_tuple(db.scan(sc, q)) == want


def test_rows_that_do_not_arrive_in_the_first_of_several_rounds():
    """40,000 query rows of a 20-letter alphabet: 8-row passes in several rounds on a cluster, which stops
    between the rounds."""
    rng = np.random.default_rng(77)
    seqs = [list(rng.integers(0, 20, n)) for n in (150, 333, 90)]
    db = (hy.Database.builder().sequences(seqs).scoring(hy.Scoring(20, BLOSUM62, 11, 1)).mode(hy.Mode.Sw)
          .search_type(hy.SearchType.ScoreEnd).max_query_len(40_000).build())
    sc = hy.Scratch(db)
    q = rng.integers(0, 20, 40_000)
    want = o.OracleDb(seqs, BLOSUM62, 20, 11, 1, 0, 1).scan(list(q))
    with _RowPolls():
        _times_out(lambda: db.scan(sc, q))
    assert hit_tuple(db.scan(sc, q)) == want
