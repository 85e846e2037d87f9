"""DIV-RF with small packets and many of them: decoders of 1 and 2 warps a packet, and the warp
decoder where 32 lanes hold a few segments of distinct values; y against the binary128 row sums,
and the time against the warp decoder asked for by name."""
import numpy as np
import pytest

from conftest import rel_row_error
from test_gpu_div_segments import TOL, _values
from test_gpu_pools import MB, _OnlyFree

pytestmark = pytest.mark.gpu

SEGMENTS, WARP = 3, 2


def _matrix(m, k, n, kind, r, lengths=None):
    lengths = np.full(m, k) if lengths is None else lengths
    rp = np.zeros(m + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    ci = (np.repeat(r.integers(0, n - lengths.max(), m), lengths) + np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)).astype(np.int32)
    return rp, ci, _values(kind, int(rp[-1]), r), r.uniform(-1, 1, n)


@pytest.mark.parametrize("kind", ["distinct", "one", "few", "mixed"])
@pytest.mark.parametrize("L,packet", [(1, 64), (4, 64), (4, 1000), (8, 300), (16, 500), (32, 64), (32, 500)])
def test_one_and_two_warps(sb, orc, L, packet, kind):
    """Uneven and empty rows, rows split over packets; the last packets incomplete."""
    r = np.random.default_rng(packet + L)
    m, n = 400 * packet // 10, 3000
    lengths = r.integers(0, 420, m)
    lengths[r.random(m) < 0.9] = r.integers(0, 40)
    lengths[11] = 2999
    rp, ci, v, x = _matrix(m, 0, n + 1, kind, r, lengths)
    h = sb.csr_to_format(rp, ci, v, m, n + 1, int(rp[-1]), format="div_rf", vec_len=L, div_packet_vals=packet)
    gold, absy = orc.csr_gold(rp, ci, v, x)
    assert rel_row_error(h.spmv(x, np.full(m, 1.0)), gold, absy) <= TOL


# packets of 8 rows, 128 distinct values (4 lanes: 256 a segment, 32 lanes: 512)
@pytest.mark.parametrize("L,packet,packets,choice", [(4, 128, 6000, (SEGMENTS, 1)), (4, 512, 1200, (SEGMENTS, 2)),
                                                     (32, 256, 6000, (SEGMENTS, 1)), (32, 1024, 1200, (SEGMENTS, 2)),
                                                     (32, 2048, 9000, (WARP, 0)), (32, 2048, 2000, (SEGMENTS, 4))])
def test_decoder_by_packets(sb, orc, L, packet, packets, choice):
    r = np.random.default_rng(packets)
    m, n = 8 * packets, 3000
    rp, ci, v, x = _matrix(m, packet // 8, n, "distinct", r)
    h = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), format="div_rf", vec_len=L, div_packet_vals=packet)
    assert h.exec_choice() == choice
    gold, absy = orc.csr_gold(rp, ci, v, x)
    assert rel_row_error(h.spmv(x, np.full(m, 1.0)), gold, absy) <= TOL


@pytest.mark.parametrize("packet", [256, 512, 1024, 2048])
def test_small_packets_are_no_slower_than_on_the_warp_decoder(sb, packet):
    """32 lanes, 12 M distinct values: within 15% of the decoder that was the default (segments of
    four warps took up to 2.6 times as long)."""
    import torch

    m, n = 600000, 600000
    rp, ci, v, _ = _matrix(m, 20, n, "distinct", np.random.default_rng(packet))
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    times = []
    for kernel in (-1, 2):
        h = sb.csr_to_format(rp, ci, v, m, n, int(rp[-1]), format="div_rf", vec_len=32, div_packet_vals=packet, kernel=kernel)
        best = float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                h.spmv(x, y)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
        h.destroy()
    assert times[0] <= 1.15 * times[1], times


@pytest.mark.parametrize("L,other", [(32, 2), (4, 0)])
def test_a_matrix_without_room_for_the_segments(sb, L, other):
    """Where the conversion fits for the decoder without segment tables, it fits for the default."""
    import torch

    m = 200000
    rp, ci, v, x = _matrix(m, 20, m, "few", np.random.default_rng(L))
    csr = [torch.from_numpy(a).cuda() for a in (rp, ci, v)]
    xd = torch.from_numpy(x).cuda()
    kw = dict(format="div_rf", vec_len=L, div_packet_vals=64)
    roomy = sb.csr_to_format(*csr, **kw)
    assert roomy.exec_choice()[0] == SEGMENTS
    roomy.destroy()
    named = sb.csr_to_format(*csr, kernel=other, **kw)
    expect, y = named.spmv(xd), torch.zeros_like(xd)
    torch.cuda.synchronize()
    named.destroy()
    for left in range(96, 1600, 32):
        sb.release_memory()
        with _OnlyFree(torch, left * MB):
            try:
                sb.csr_to_format(*csr, kernel=other, **kw).destroy()
            except sb.SpmvError as e:
                assert e.status == sb._capi.SPMV_ERR_NOMEM
                continue
            sb.release_memory()
            h = sb.csr_to_format(*csr, **kw)
            choice = h.exec_choice()
            h.spmv(xd, y)
            h.destroy()
            sb.release_memory()
            break
    assert choice == (other, 0)
    assert torch.allclose(y, expect, rtol=1e-12, atol=1e-12)
