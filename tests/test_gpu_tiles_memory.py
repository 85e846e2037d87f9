"""Row tiles and device memory: a layout that is refused leaves nothing allocated, and one that finds
no memory leaves the matrix to the kernels that need no copy of its entries."""
import numpy as np
import pytest

from test_gpu_pools import MB, _device_matrix, _OnlyFree
from test_gpu_tiles import FORMS, N, THRESHOLD, _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,kw", [(f, kw) for f, kw in FORMS if kw.get("vec_len", 1) <= 8 and f in ("csr_naive", "csr_vec", "sell")])
def test_a_refused_layout_keeps_no_memory(sb, fmt, kw):
    """A row of 31 among rows of one entry in every window: its slice alone would double the stored
    entries, so the matrix holds what it holds on the kernel that then runs."""
    m = 3420 * 1024 + 5
    lengths = np.full(m, 1)
    lengths[::1024] = 31
    rp, ci, v, _ = _matrix(lengths, 3)
    args = (rp, ci, v, m, N, int(rp[-1]))
    assert rp[-1] >= THRESHOLD
    h = sb.csr_to_format(*args, format=fmt, **kw)
    assert h.exec_choice() == (4, 0)
    assert h.device_bytes == sb.csr_to_format(*args, format=fmt, kernel=4, **kw).device_bytes


@pytest.mark.parametrize("fmt,kw,kernel", [("csr_naive", {}, 4), ("csr_vec", dict(vec_len=4), 4), ("sell", dict(vec_len=4), 4),
                                           ("sell_c_s", {}, 10), ("csr_naive", dict(value_type="f32"), 4)])
def test_a_matrix_without_room_for_the_layout(sb, fmt, kw, kernel):
    """With the least memory (to 32 MB) that the conversion for a staged kernel takes, the default has no
    room for a layout of 240 MB (FP32: 160) beside it, and runs that kernel.  (sell_sorted: the
    scratch of its reordering is as large, so the layout always finds its place.)"""
    import torch

    csr = _device_matrix(torch, 20_000_000, 400000)
    x = torch.rand(400000, dtype=torch.float64, device="cuda")
    if "value_type" in kw:
        x = x.float()
    roomy = sb.csr_to_format(*csr, format=fmt, **kw)
    assert roomy.exec_choice()[0] == 11
    expect, y = roomy.spmv(x), torch.zeros_like(x)
    roomy.destroy()
    for left in range(256, 1024, 32):
        sb.release_memory()
        with _OnlyFree(torch, left * MB):
            try:
                sb.csr_to_format(*csr, format=fmt, kernel=kernel, **kw).destroy()
            except sb.SpmvError as e:
                assert e.status == sb._capi.SPMV_ERR_NOMEM
                continue
            sb.release_memory()
            h = sb.csr_to_format(*csr, format=fmt, **kw)
            choice = h.exec_choice()
            h.spmv(x, y)
            h.destroy()
            sb.release_memory()
            break
    assert choice == (kernel, 0)
    assert torch.equal(y, expect)


def test_a_batch_without_room_for_the_layout(sb):
    import torch

    k = 100
    m = 100000
    rp = np.arange(m + 1, dtype=np.int32) * k
    r = np.random.default_rng(5)
    mats = [(rp, (np.tile(np.arange(k), m) + np.repeat(r.integers(0, m - k, m), k)).astype(np.int32), r.uniform(-1, 1, k * m), m, m)
            for _ in range(2)]
    x = torch.rand(2 * m, dtype=torch.float64, device="cuda")
    roomy = sb.Batch(mats, ["sell", "csr_naive"])
    expect, y = torch.zeros_like(x), torch.zeros_like(x)
    roomy.spmv(x, expect)
    roomy.sync()
    roomy.destroy()
    sb.release_memory()
    with _OnlyFree(torch, 500 * MB):                     # 360 MB of arrays, 240 of the layout
        b = sb.Batch(mats, ["sell", "csr_naive"])
        b.spmv(x, y)
        b.sync()
        b.destroy()
        sb.release_memory()
    assert torch.equal(y, expect)
