"""Which kernels the default descriptors run: the matrices that the tests of row tiles and of the
segment decoder use do reach the builds that those tests are named for."""
import numpy as np
import pytest

from conftest import rel_row_error
from test_gpu_tiles import FORMS, LARGE, N, _matrix
from test_gpu_tiles_wide import N as WIDE_N
from test_gpu_tiles_wide import _case

pytestmark = pytest.mark.gpu

TILES, WIDE, STAGED = 11, 1, 2


@pytest.mark.parametrize("paired", [True, False])
@pytest.mark.parametrize("fmt,kw", FORMS + [("csr_naive", dict(value_type="f32"))])
def test_builds_of_large_matrices(sb, fmt, kw, paired):
    """Rows that share columns take the build that fetches their lines once; csr_vec and FP32 have none."""
    rp, ci, v, _ = _case(paired)
    shared = paired and fmt != "csr_vec" and "value_type" not in kw
    h = sb.csr_to_format(rp, ci, v, rp.size - 1, WIDE_N, int(rp[-1]), format=fmt, **kw)
    assert h.exec_choice() == (TILES, WIDE + (STAGED if shared else 0))


@pytest.mark.parametrize("fmt,kw", FORMS)
def test_builds_of_smaller_matrices(sb, fmt, kw):
    rp, ci, v, _ = _matrix(np.full(LARGE // 12, 12), 12)
    h = sb.csr_to_format(rp, ci, v, rp.size - 1, N, int(rp[-1]), format=fmt, **kw)
    assert h.exec_choice() == (TILES, 0)


def test_named_kernels_are_what_runs(sb):
    rp, ci, v, _ = _matrix(np.full(2000, 12), 1)
    for fmt, kernel in [("csr_naive", 4), ("csr_naive", 0), ("sell", 2), ("sell_c_s", 10), ("div_rf", 0)]:
        h = sb.csr_to_format(rp, ci, v, 2000, N, int(rp[-1]), format=fmt, kernel=kernel)
        assert h.exec_choice() == (kernel, 0), fmt


def test_batches(sb):
    rp, ci, v, _ = _matrix(np.full(2000, 12), 1)
    mats = [(rp, ci, v, 2000, N)] * 2
    assert sb.Batch(mats, ["sell", "csr_naive"]).exec_choice() == (TILES, 0)
    assert sb.Batch(mats, [dict(format=f, block_nnz=512) for f in ("sell", "csr_naive")]).exec_choice() == (0, 0)
    assert sb.Batch(mats, ["csr_naive", "csr_naive"]).exec_choice() == (4, 0)


@pytest.mark.parametrize("packets,choice", [(100, 32), (250, 16), (400, 8 + 64), (500, 8), (800, 4)])
@pytest.mark.parametrize("L", [4, 32])
def test_warps_a_packet(sb, orc, L, packets, choice):
    """Packets of 8 rows of distinct values, four segments each."""
    r = np.random.default_rng(packets)
    k = 128 if L == 4 else 256                           # segments of 256 and 512
    m, n = 8 * packets, 3000
    rp = (np.arange(m + 1) * k).astype(np.int32)
    ci = (np.repeat(r.integers(0, n - k, m), k) + np.tile(np.arange(k), m)).astype(np.int32)
    v, x = r.integers(-(1 << 30), 1 << 30, k * m) / (1 << 30), r.uniform(-1, 1, n)
    h = sb.csr_to_format(rp, ci, v, m, n, k * m, format="div_rf", vec_len=L, div_packet_vals=8 * k)
    assert h.exec_choice() == (3, choice)
    gold, absy = orc.csr_gold(rp, ci, v, x)
    assert rel_row_error(h.spmv(x, np.full(m, 1.0)), gold, absy) <= 1e-12
