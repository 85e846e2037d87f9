"""Overlapped launches in a loop take no longer than launches that a kernel between them keeps apart."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _per_step(torch, steps, step):
    best = float("inf")
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(steps):
            step()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) / steps)
    return best


@pytest.mark.parametrize("C,rows,width", [(64, 16554, 45), (64, 60000, 20), (128, 20000, 40), (32, 16554, 45)])
def test_tiled_slices(sb, C, rows, width):
    """SELL-C-sigma on kernel 8: few long blocks a CTA (1.2 to 1.4 times as long overlapped before)."""
    import torch

    r = np.random.default_rng(rows)
    lengths = np.maximum(0, r.normal(width, width / 8, rows)).astype(np.int64)
    rp = np.zeros(rows + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    ci = np.sort(r.integers(0, rows, (rows, int(lengths.max()))), axis=1).astype(np.int32)
    ci = ci[np.arange(ci.shape[1]) < lengths[:, None]]
    x = torch.rand(rows, dtype=torch.float64, device="cuda")
    y, flag = torch.empty_like(x), torch.zeros(1, device="cuda")
    h = sb.csr_to_format(rp, ci, r.uniform(-1, 1, rp[-1]), format="sell_c_s", sellcs_c=C, sellcs_sigma=8 * C, kernel=8)

    def apart():
        h.spmv(x, y)
        flag.fill_(1.0)

    assert _per_step(torch, 400, lambda: h.spmv(x, y)) <= _per_step(torch, 400, apart)
