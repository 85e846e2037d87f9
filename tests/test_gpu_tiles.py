"""Row tiles, the default execution layout of larger matrices: y bit for bit against the oracle's
restatement of each format at the edges of the layout (windows of 1,024 rows, slices of 32,
tiles of 8 columns, rows summed by a warp of their own in steps of 256 entries), and against the
general staged kernel where x holds infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


N = 5000
THRESHOLD = 3500000      # entries from which the default is row tiles
LARGE = 3600000


def _matrix(lengths, seed, n=N):
    """CSR with the given row lengths: columns from a random start, 1 to 3 apart."""
    r = np.random.default_rng(seed)
    lengths = np.asarray(lengths, np.int64)
    rp = np.zeros(lengths.size + 1, np.int64)
    np.cumsum(lengths, out=rp[1:])
    step = np.minimum(r.integers(1, 4, lengths.size), np.maximum(1, n // np.maximum(lengths, 1)))
    start = (r.random(lengths.size) * (n - step * lengths + 1)).astype(np.int64)
    k = np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)
    ci = np.repeat(start, lengths) + k * np.repeat(step, lengths)
    return rp.astype(np.int32), ci.astype(np.int32), r.uniform(-1, 1, rp[-1]), r.uniform(-1, 1, n)


def _bits_equal(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint64), np.ascontiguousarray(b).view(np.uint64))


FORMS = [("csr_naive", {}), ("csr_vec", dict(vec_len=4)), ("csr_vec", dict(vec_len=8)), ("sell", dict(vec_len=4)),
         ("sell", dict(vec_len=16)), ("sell_sorted", dict(vec_len=4)), ("sell_sorted", dict(vec_len=32)),
         ("sell_c_s", dict(sellcs_c=32, sellcs_sigma=512)), ("sell_c_s", dict(sellcs_c=64, sellcs_sigma=128))]


def _expected(orc, fmt, kw, rp, ci, v, x):
    m = rp.size - 1
    if fmt == "csr_naive":
        return orc.csr_spmv(rp, ci, v, x)
    if fmt == "csr_vec":
        return orc.csr_vec_spmv(rp, ci, v, x, kw["vec_len"])
    if fmt == "sell":
        return orc.sell_spmv(orc.sell_convert(rp, ci, v, kw["vec_len"], 8), m, kw["vec_len"], x)
    if fmt == "sell_sorted":
        return orc.sell_sorted_spmv(orc.sell_sorted_convert(rp, ci, v, kw["vec_len"], 8), m, kw["vec_len"], x)
    return orc.sellcs_spmv(orc.sellcs_convert(rp, ci, v, kw["sellcs_c"], kw["sellcs_sigma"]), m, kw["sellcs_c"], x)


@pytest.mark.parametrize("fmt,kw", FORMS)
@pytest.mark.parametrize("rest", [0, 1, 31, 33, 1023])
def test_edges_of_rows_and_tiles(sb, orc, fmt, kw, rest):
    m = 190 * 1024 + rest
    r = np.random.default_rng(rest)
    lengths = r.integers(0, 39, m)
    lengths[r.random(m) < 0.05] = 0                       # empty rows
    for i, k in enumerate([255, 256, 257, 511, 513, 7, 8, 9, 64, 1030]):
        lengths[(3701 * i + 5) % m] = k                   # rows of a warp of their own, whole tiles
    rp, ci, v, x = _matrix(lengths, rest)
    assert rp[-1] >= THRESHOLD
    y = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format=fmt, **kw).spmv(x, np.full(m, 1.0))
    assert _bits_equal(y, _expected(orc, fmt, kw, rp, ci, v, x))


@pytest.mark.parametrize("m,longest", [(1, 40), (31, 9), (33, 300), (1025, 64), (2050, 1030)])
@pytest.mark.parametrize("C,sigma", [(32, 512), (64, 128)])
def test_small_sell_c_sigma(sb, orc, C, sigma, m, longest):
    r = np.random.default_rng(m)
    lengths = r.integers(0, 27, m)
    lengths[m // 2] = longest
    rp, ci, v, x = _matrix(lengths, m)
    kw = dict(sellcs_c=C, sellcs_sigma=sigma)
    y = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format="sell_c_s", **kw).spmv(x, np.full(m, 1.0))
    assert _bits_equal(y, _expected(orc, "sell_c_s", kw, rp, ci, v, x))


@pytest.mark.parametrize("width", [1, 3, 8, 12, 21, 32, 47])
@pytest.mark.parametrize("fmt,kw", FORMS)
def test_equal_rows_of_every_remainder(sb, orc, fmt, kw, width):
    """Whole slices of one width: every kind of last tile."""
    m = LARGE // width + 7
    rp, ci, v, x = _matrix(np.full(m, width), width)
    y = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format=fmt, **kw).spmv(x, np.full(m, 1.0))
    assert _bits_equal(y, _expected(orc, fmt, kw, rp, ci, v, x))


@pytest.mark.parametrize("fmt,kw", FORMS)
def test_padding_heavy_matrix_keeps_the_staged_kernels(sb, orc, fmt, kw):
    """One longer row among short ones in every window: the layout would store far more than
    the entries, so the matrix stays on the staged kernels."""
    m = 1800 * 1024 + 5
    lengths = np.full(m, 2)
    lengths[::1024] = 60
    rp, ci, v, x = _matrix(lengths, 3)
    y = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format=fmt, **kw).spmv(x, np.full(m, 1.0))
    assert _bits_equal(y, _expected(orc, fmt, kw, rp, ci, v, x))


@pytest.mark.parametrize("fmt,kw", FORMS)
def test_infinities_and_nan_as_the_general_kernel(sb, fmt, kw):
    m = 180 * 1024
    r = np.random.default_rng(8)
    lengths = r.integers(0, 42, m)
    lengths[17] = 600
    rp, ci, v, x = _matrix(lengths, 5)
    x[::97] = np.inf
    x[3::111] = -np.inf
    x[5::213] = np.nan
    x[0] = np.inf                                         # SELL-C-sigma pads with column 0
    y = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format=fmt, **kw).spmv(x)
    ref = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format=fmt, kernel=0, **kw).spmv(x)
    assert np.array_equal(np.isnan(y), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert ok.any() and _bits_equal(y[ok], ref[ok])


@pytest.mark.parametrize("rest", [0, 1, 33])
def test_fp32_rows(sb, orc, rest):
    """The FP32 variant on row tiles: the sequential Dot2 rows bit for bit."""
    m = 190 * 1024 + rest
    r = np.random.default_rng(100 + rest)
    lengths = r.integers(0, 39, m)
    for i, k in enumerate([0, 255, 256, 257, 600, 8, 9, 64]):
        lengths[(3701 * i + 5) % m] = k
    rp, ci, v, x = _matrix(lengths, rest)
    assert rp[-1] >= THRESHOLD
    x32 = x.astype(np.float32)
    mf = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format="csr_naive", value_type="f32")
    y = mf.spmv(x32, np.full(m, 1.0, np.float32))
    assert np.array_equal(y.view(np.uint32), orc.csr_f32_dot2(rp, ci, v.astype(np.float32), x32).view(np.uint32))


def test_batch_of_edges(sb, orc):
    """A mixed batch: empty and one-row matrices, sizes around slices and windows, long rows."""
    import torch

    r = np.random.default_rng(21)
    mats, fmts = [], []
    for i, m in enumerate([1, 0, 33, 1024, 1025, 2050, 5000, 31, 64, 3000, 7, 4097]):
        lengths = r.integers(0, 60, m)
        if m:
            lengths[m // 2] = 300 + 211 * i
        rp, ci, v, x = _matrix(lengths, i)
        mats.append((rp, ci, v, m, N))
        fmts.append([("csr_naive", {}), ("sell", dict(vec_len=4)), ("sell_sorted", dict(vec_len=8)),
                     ("sell_c_s", dict(sellcs_c=32, sellcs_sigma=512))][i % 4])
    b = sb.Batch(mats, [dict(kw, format=f) for f, kw in fmts])
    x = r.uniform(-1, 1, b.total_x)
    yd = torch.full((b.total_y,), 5.0, dtype=torch.float64, device="cuda")
    b.spmv(torch.from_numpy(x).cuda(), yd)
    b.sync()
    y = yd.cpu().numpy()
    for (rp, ci, v, m, n), (f, kw), xo, yo in zip(mats, fmts, b.x_offsets, b.y_offsets):
        if m:
            assert _bits_equal(y[yo:yo + m], _expected(orc, f, kw, rp, ci, v, x[xo:xo + n])), (m, f)
