"""The library's memory pools: what they keep between conversions, and what they give back."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(r, m):
    lengths = r.integers(0, 30, m)
    rp = np.zeros(m + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    ci = (np.repeat(r.integers(0, m - 64, m), lengths) + np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)).astype(np.int32)
    return rp, ci, r.uniform(-1, 1, rp[-1]), m, m


def test_conversion_time_does_not_grow_with_the_matrices_alive(sb):
    """A batch of 48 uneven matrices beside four others alive: no more than twice the time it takes
    beside none (four to five times while every allocation asked all their streams)."""
    r = np.random.default_rng(1)
    mats = [_matrix(r, int(1000 * 100 ** u)) for u in r.random(48)]
    fmts = ["sell", "sell_sorted", "sell_c_s", "csr_naive"] * 12

    def least():
        best = float("inf")
        for _ in range(5):
            t = time.perf_counter()
            b = sb.Batch(mats, fmts)
            best = min(best, time.perf_counter() - t)
            del b
        return best

    alone = least()
    alive = [sb.Batch(mats, fmts) for _ in range(4)]
    beside = least()
    assert len(alive) == 4 and beside < 2 * alone, (alone, beside)
