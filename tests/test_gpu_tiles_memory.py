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


# what is left free (MB): the format's arrays of 20 M entries fit, the layout's 240 (FP32: 160) beside them do not
@pytest.mark.parametrize("fmt,kw,left", [("csr_naive", {}, 400), ("csr_vec", dict(vec_len=4), 400),
                                         ("sell", dict(vec_len=4), 640), ("sell_sorted", dict(vec_len=8), 740),
                                         ("sell_c_s", {}, 660), ("csr_naive", dict(value_type="f32"), 420)])
def test_a_matrix_without_room_for_the_layout(sb, fmt, kw, left):
    import torch

    csr = _device_matrix(torch, 20_000_000)
    x = torch.rand(100000, dtype=torch.float64, device="cuda")
    if "value_type" in kw:
        x = x.float()
    roomy = sb.csr_to_format(*csr, format=fmt, **kw)
    expect, y, roomy_bytes = roomy.spmv(x), torch.zeros_like(x), roomy.device_bytes
    roomy.destroy()
    sb.release_memory()
    with _OnlyFree(torch, left * MB):
        h = sb.csr_to_format(*csr, format=fmt, **kw)
        h.spmv(x, y)
        tight_bytes = h.device_bytes
        h.destroy()
        sb.release_memory()
    assert roomy_bytes - tight_bytes >= (80 if fmt == "sell_c_s" else 150) * MB      # the layout was there, and is not
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
