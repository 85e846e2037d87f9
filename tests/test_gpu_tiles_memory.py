"""Row tiles and device memory: a layout that is refused leaves nothing allocated."""
import numpy as np
import pytest

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
    assert sb.csr_to_format(*args, format=fmt, **kw).device_bytes == \
        sb.csr_to_format(*args, format=fmt, kernel=4, **kw).device_bytes
