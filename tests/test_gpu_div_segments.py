"""DIV-RF's segment decoder (the default up to 32 lanes) against the CTA decoder and the
binary128 row sums: groups of every kind (whole positions, an incomplete one, coordinates of one
value split over segments), every lane count, packets of few and many values."""
import numpy as np
import pytest

from conftest import rel_row_error

pytestmark = pytest.mark.gpu

TOL = 1e-12      # per row, relative to max(|y|, sum |a x|): the bound of every DIV-RF sum


def _values(kind, nnz, r):
    if kind == "distinct":
        return r.integers(-(1 << 30), 1 << 30, nnz) / (1 << 30)
    if kind == "one":
        return np.full(nnz, 0.37)
    if kind == "few":
        return r.uniform(-1, 1, 40)[(r.random(nnz) ** 2 * 40).astype(int)]
    v = r.uniform(-1, 1, nnz)                            # mixed: half distinct, half from few
    few = r.uniform(-1, 1, 7)
    pick = r.random(nnz) < 0.5
    v[pick] = few[r.integers(0, 7, int(pick.sum()))]
    v[r.random(nnz) < 0.02] = 0.0
    return v


@pytest.mark.parametrize("L", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("packet", [64, 1000, 16384])
@pytest.mark.parametrize("kind", ["distinct", "one", "few", "mixed"])
def test_segments_match_the_cta_decoder(sb, orc, kind, packet, L):
    r = np.random.default_rng(L * 7 + packet)
    m, n = 1500, 900
    lengths = r.integers(0, 40, m)
    lengths[7], lengths[800] = 900, 333                  # rows split across packets
    rp = np.zeros(m + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    ci = np.concatenate([np.sort(r.choice(n, k, replace=False)) for k in lengths]).astype(np.int32)
    v, x = _values(kind, int(rp[-1]), r), r.uniform(-1, 1, n)
    kw = dict(format="div_rf", vec_len=L, div_packet_vals=packet)
    y = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), **kw).spmv(x, np.full(m, 1.0))
    y0 = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), kernel=0, **kw).spmv(x, np.full(m, 1.0))
    gold, absy = orc.csr_gold(rp, ci, v, x)
    assert rel_row_error(y, gold, absy) <= TOL
    assert rel_row_error(y, y0, absy) <= TOL


@pytest.mark.parametrize("packets", [100, 200, 400, 1500])
@pytest.mark.parametrize("L", [4, 32])
def test_long_rows_and_every_packet_width(sb, orc, L, packets):
    """4 to 32 warps a packet by their number; packets of one long row and of many short ones."""
    r = np.random.default_rng(packets + L)
    n = 3000
    lengths = r.integers(0, 5, packets * 16)
    lengths[:packets // 100] = n                         # packets of one row: 32 sums a row
    rp = np.zeros(len(lengths) + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    ci = np.concatenate([np.sort(r.choice(n, k, replace=False)) for k in lengths]).astype(np.int32)
    m, nnz = len(lengths), int(rp[-1])
    v, x = _values("mixed", nnz, r), r.uniform(-1, 1, n)
    y = sb.csr_to_format(rp, ci, v, m, n, nnz, format="div_rf", vec_len=L, div_packet_vals=64).spmv(x, np.full(m, 1.0))
    gold, absy = orc.csr_gold(rp, ci, v, x)
    assert rel_row_error(y, gold, absy) <= TOL
