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


def _handle(sb, torch, rows, width, fmt, **kw):
    """Even rows with columns far apart; an SpMV to call."""
    r = np.random.default_rng(rows)
    rp = (np.arange(rows + 1) * width).astype(np.int32)
    ci = (r.integers(0, rows - 8 * width, rows)[:, None] + 8 * np.arange(width)).astype(np.int32).ravel()
    h = sb.csr_to_format(rp, ci, r.uniform(-1, 1, rows * width), format=fmt, **kw)
    x = torch.rand(rows, dtype=torch.float32 if "value_type" in kw else torch.float64, device="cuda")
    y = torch.empty_like(x)
    return h, lambda: h.spmv(x, y)


TILES, STAGED, FEW = (300000, 24, "sell", dict(vec_len=4)), (40000, 45, "sell_c_s", {}), (2000, 20, "csr_naive", {})
FP32, DIV = (100000, 20, "csr_naive", dict(value_type="f32")), (100000, 24, "div_rf", {})


@pytest.mark.parametrize("order", [(TILES, STAGED), (TILES, FP32), (STAGED, DIV), (TILES, FEW), (TILES, FEW, STAGED), (STAGED, FEW, FEW, TILES)])
def test_kernels_by_turns(sb, order):
    """Kernels of different shared memory in turn (up to 1.9 times as long overlapped before)."""
    import torch

    steps = [_handle(sb, torch, rows, width, fmt, **kw) for rows, width, fmt, kw in order]
    flag = torch.zeros(1, device="cuda")

    def together():
        for _, step in steps:
            step()

    def apart():
        for _, step in steps:
            step()
            flag.fill_(1.0)

    assert _per_step(torch, 100, together) <= _per_step(torch, 100, apart)


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
