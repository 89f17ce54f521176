"""align_pairs whose long pairs' stripes give up (every bounded wait runs out at once) while the chunks' other
kernels are still on their streams: the failed call returns with none of its work left on the device, and the
next call's results are the oracle's."""
import numpy as np
import pytest

import hyalite_b200 as hy
import pyoracle as o
from conftest import DNA
from hyalite_b200 import _abi

pytestmark = pytest.mark.gpu


def _pairs(rng, n, long_at):
    """n pairs of 150 x 400, at long_at two of 1,100 x 1,100 (stripes)."""
    ql, tl = np.full(n, 150), np.full(n, 400)
    ql[long_at], tl[long_at] = 1100, 1100
    q_off, t_off = np.zeros(n + 1, np.uint64), np.zeros(n + 1, np.uint64)
    q_off[1:], t_off[1:] = np.cumsum(ql), np.cumsum(tl)
    q, t = rng.integers(0, 4, int(q_off[-1])), rng.integers(0, 4, int(t_off[-1]))
    return q.astype(np.uint8), q_off, t.astype(np.uint8), t_off


@pytest.mark.parametrize("n", [3000, 120_000])
def test_a_call_that_times_out_leaves_no_work_behind(n):
    rng = np.random.default_rng(n)
    sc = hy.Scoring(4, DNA, 6, 1)
    run = lambda p: hy.align_pairs_arrays(*p, sc, hy.Mode.Hw, hy.SearchType.ScoreEnd)  # noqa: E731
    run(_pairs(rng, n, [5, n - 1]))  # the buffers are grown
    for _ in range(3):
        bad, good = _pairs(rng, n, [5, n - 1]), _pairs(rng, n, [0, n // 2])
        _abi.lib.hy_debug_set_wait_polls(0)
        try:
            _, (err, _) = run(bad)
            idle = _abi.lib.hy_debug_pairs_idle()
        finally:
            _abi.lib.hy_debug_set_wait_polls(-1)
        assert err.kind == "Timeout" and idle == 1
        hits, (err, _) = run(good)
        assert err is None
        q, qo, t, to = good
        for k in [0, 1, 5, n // 2, n - 1] + [int(x) for x in rng.integers(0, n, 40)]:
            want = o.align_pair(list(q[qo[k]:qo[k + 1]]), list(t[to[k]:to[k + 1]]), DNA, 4, 6, 1, int(hy.Mode.Hw))
            assert (hits[k].score, hits[k].query_end, hits[k].target_end) == want, k
