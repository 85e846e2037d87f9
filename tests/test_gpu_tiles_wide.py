"""Row tiles above the size where the kernels of many ranges a warp take over (about 29 M entries
and slices): y bit for bit against the oracle for every format, on rows that share columns in
pairs (x is then fetched a line once for both) and on rows that share none."""
import numpy as np
import pytest

from test_gpu_tiles import FORMS, _bits_equal, _expected

pytestmark = pytest.mark.gpu

N = 6000
WIDE = 4 * 148 * 12 * 2 * 2048      # entries + 128 a slice of 32 rows, 148 SMs


def _wide_matrix(paired, seed):
    """An odd number of rows of 0 to 62 entries, slices without entries, rows of a warp of their
    own; entries of a row 40 to 90 columns apart, each in a line of its own."""
    r = np.random.default_rng(seed)
    m = 1000003
    lengths = r.integers(18, 49, m)
    lengths[r.random(m) < 0.02] = 0
    lengths[5000:7100] = 0                               # whole windows of empty rows
    lengths[::997] = 62
    step = r.integers(40, 91, m)
    for i, k in enumerate([2049, 600, 1025, 513]):       # long rows, columns 1 or 2 apart
        lengths[77777 + 111111 * i] = k
        step[77777 + 111111 * i] = 1 + i % 2
    start = (r.random(m) * (N - step * lengths)).astype(np.int64)
    if paired:                                           # every odd row has the columns of the row before it
        for a in (lengths, step, start):
            a[1::2] = a[:-1:2]
    rp = np.zeros(m + 1, np.int64)
    np.cumsum(lengths, out=rp[1:])
    k = np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)
    ci = np.repeat(start, lengths) + k * np.repeat(step, lengths)
    assert rp[-1] + m // 32 * 128 > WIDE
    return rp.astype(np.int32), ci.astype(np.int32), r.uniform(-1, 1, rp[-1]), r.uniform(-1, 1, N)


_kept = {}


def _case(paired):
    if paired not in _kept:
        _kept.clear()
        _kept[paired] = _wide_matrix(paired, 17)
    return _kept[paired]


@pytest.mark.parametrize("paired", [True, False])
@pytest.mark.parametrize("fmt,kw", FORMS)
def test_large_matrices_bit_for_bit(sb, orc, fmt, kw, paired):
    rp, ci, v, x = _case(paired)
    m = rp.size - 1
    y = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format=fmt, **kw).spmv(x, np.full(m, 1.0))
    assert _bits_equal(y, _expected(orc, fmt, kw, rp, ci, v, x))


def test_large_fp32_rows(sb, orc):
    rp, ci, v, x = _case(True)
    m = rp.size - 1
    x32 = x.astype(np.float32)
    mf = sb.csr_to_format(rp, ci, v, m, N, int(rp[-1]), format="csr_naive", value_type="f32")
    y = mf.spmv(x32, np.full(m, 1.0, np.float32))
    assert np.array_equal(y.view(np.uint32), orc.csr_f32_dot2(rp, ci, v.astype(np.float32), x32).view(np.uint32))


def test_large_mixed_batch(sb, orc):
    import torch

    rp, ci, v, x1 = _case(True)
    mats, fmts, cuts = [], [], [0, 250001, 250002, 500000, 760033, 1000003]
    for i, (a, b) in enumerate(zip(cuts[:-1], cuts[1:])):
        e0, e1 = int(rp[a]), int(rp[b])
        mats.append((rp[a:b + 1] - rp[a], ci[e0:e1], v[e0:e1], b - a, N))
        fmts.append([("csr_naive", {}), ("sell", dict(vec_len=4)), ("sell_sorted", dict(vec_len=8)),
                     ("sell_c_s", dict(sellcs_c=32, sellcs_sigma=512))][i % 4])
    b = sb.Batch(mats, [dict(kw, format=f) for f, kw in fmts])
    x = np.random.default_rng(4).uniform(-1, 1, b.total_x)
    yd = torch.full((b.total_y,), 5.0, dtype=torch.float64, device="cuda")
    b.spmv(torch.from_numpy(x).cuda(), yd)
    b.sync()
    y = yd.cpu().numpy()
    for (p, c, w, m, n), (f, kw), xo, yo in zip(mats, fmts, b.x_offsets, b.y_offsets):
        assert _bits_equal(y[yo:yo + m], _expected(orc, f, kw, p, c, w, x[xo:xo + n])), (m, f)
