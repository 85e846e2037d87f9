"""Row tiles or kernel 4: few long rows run kernel 4, which is the faster there, rows enough for the
chip run row tiles; y bit for bit against the oracle on either side, and the default's time against
the kernels asked for by name."""
import numpy as np
import pytest

from test_gpu_tiles import FORMS, _bits_equal, _expected

pytestmark = pytest.mark.gpu

SHAPES = [(2000, 2000), (6000, 620), (20000, 200), (40003, 100)]


def _even(m, k, n, seed):
    """Rows of k - 2 to k + 2 entries, 20 to 27 columns apart: a line of x each."""
    r = np.random.default_rng(seed)
    lengths = r.integers(k - 2, k + 3, m)
    rp = np.zeros(m + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    step = r.integers(20, 28, m)
    start = (r.random(m) * (n - step * lengths)).astype(np.int64)
    at = np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)
    ci = (np.repeat(start, lengths) + at * np.repeat(step, lengths)).astype(np.int32)
    return rp, ci, r.uniform(-1, 1, rp[-1]), r.uniform(-1, 1, n)


@pytest.mark.parametrize("m,k", SHAPES)
@pytest.mark.parametrize("fmt,kw", FORMS)
def test_few_long_rows(sb, orc, fmt, kw, m, k):
    n = 28 * (k + 3)
    rp, ci, v, x = _even(m, k, n, k)
    h = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), format=fmt, **kw)
    # csr_vec: kernel 4 sums rows above its blocks in few threads, and 8 lanes differ little with rows of 100
    if fmt != "csr_vec" or 100 < k < 1000:
        assert h.exec_choice() == (4, 0)
    assert _bits_equal(h.spmv(x, np.full(m, 1.0)), _expected(orc, fmt, kw, rp, ci, v, x))


@pytest.mark.parametrize("fmt,kw", [("sell", dict(vec_len=32)), ("sell_sorted", dict(vec_len=32)), ("sell_c_s", {})])
def test_long_even_rows_in_slices_of_32(sb, orc, fmt, kw):
    m, k = 60003, 200
    n = 28 * (k + 3)
    rp, ci, v, x = _even(m, k, n, k)
    h = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), format=fmt, **kw)
    assert h.exec_choice() == (10, 0)
    if fmt == "sell_c_s":
        kw = dict(sellcs_c=32, sellcs_sigma=512)
    assert _bits_equal(h.spmv(x, np.full(m, 1.0)), _expected(orc, fmt, kw, rp, ci, v, x))


@pytest.mark.parametrize("fmt,kw", [f for f in FORMS if f[0] != "csr_naive"])
def test_many_longer_rows(sb, orc, fmt, kw):
    """Exponential lengths: thousands of rows above the first bound of rows with a warp of their own."""
    r = np.random.default_rng(11)
    m, n = 700003, 30000
    lengths = r.exponential(14.0, m).astype(np.int64)
    rp = np.zeros(m + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    start = (r.random(m) * (n - 20 * lengths)).astype(np.int64)
    ci = (np.repeat(start, lengths) + 20 * (np.arange(rp[-1]) - np.repeat(rp[:-1], lengths))).astype(np.int32)
    v, x = r.uniform(-1, 1, rp[-1]), r.uniform(-1, 1, n)
    h = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), format=fmt, **kw)
    assert h.exec_choice()[0] == 11
    assert _bits_equal(h.spmv(x, np.full(m, 1.0)), _expected(orc, fmt, kw, rp, ci, v, x))


@pytest.mark.parametrize("m,k", [(2000001, 5), (600000, 9)])
def test_short_rows_of_csr_naive(sb, orc, m, k):
    """Kernel 4 at any size (row tiles took 1.1 to 1.2 times as long)."""
    rp, ci, v, x = _even(m, k, 28 * (k + 3), k)
    args = (rp, ci, v, m, x.size, int(rp[-1]))
    h, named = sb.csr_to_format(*args, format="csr_naive"), sb.csr_to_format(*args, format="csr_naive", kernel=4)
    assert h.exec_choice() == (4, 0)
    assert h.device_bytes == named.device_bytes
    assert _bits_equal(h.spmv(x, np.full(m, 1.0)), orc.csr_spmv(rp, ci, v, x))


@pytest.mark.parametrize("k", [21, 32, 47])
@pytest.mark.parametrize("fmt,kw", FORMS)
def test_rows_enough_for_the_chip(sb, orc, fmt, kw, k):
    m = 190001
    n = 28 * (k + 3)
    rp, ci, v, x = _even(m, k, n, k)
    h = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), format=fmt, **kw)
    assert h.exec_choice() == (11, 0)
    assert _bits_equal(h.spmv(x, np.full(m, 1.0)), _expected(orc, fmt, kw, rp, ci, v, x))


@pytest.mark.parametrize("m,k", SHAPES + [(16554, 45), (100001, 45), (60003, 200), (200001, 200)])
@pytest.mark.parametrize("fmt,kw,kernels", [("csr_naive", {}, (4,)), ("csr_naive", dict(value_type="f32"), (4,)),
                                            ("csr_vec", dict(vec_len=4), (4,)), ("sell", dict(vec_len=4), (4,)),
                                            ("sell_sorted", dict(vec_len=32), (10,)),
                                            ("sell_c_s", {}, (4, 10)), ("sell_c_s", dict(sellcs_c=64, sellcs_sigma=1024), (4, 8))])
def test_default_is_near_the_fastest(sb, fmt, kw, kernels, m, k):
    """Within a quarter and 1 us of the kernels asked for by name (up to 8 times as long before)."""
    import torch

    n = 28 * (k + 3)
    rp, ci, v, x = _even(m, k, n, k)
    xd = torch.from_numpy(x.astype(np.float32 if "value_type" in kw else np.float64)).cuda()
    y = torch.zeros(m, dtype=xd.dtype, device="cuda")
    times = []
    for kernel in (-1,) + kernels:
        h = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), format=fmt, kernel=kernel, **kw)
        best = float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(100):
                h.spmv(xd, y)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 10)
        times.append(best)
        h.destroy()
    assert times[0] <= 1.25 * min(times[1:]) + 1.0, times
