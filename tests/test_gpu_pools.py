"""The library's memory pools: what they keep between conversions, and what they give back."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20
KEEP = 512 * MB          # unused memory a pool keeps


def _matrix(r, m):
    lengths = r.integers(0, 30, m)
    rp = np.zeros(m + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    ci = (np.repeat(r.integers(0, m - 64, m), lengths) + np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)).astype(np.int32)
    return rp, ci, r.uniform(-1, 1, rp[-1]), m, m


def test_conversion_time_does_not_grow_with_the_matrices_alive(sb):
    """A batch of 48 uneven matrices beside four others alive: no more than twice the time it takes
    beside none (four to five times while every allocation asked all their streams)."""
    r = np.random.default_rng(1)
    mats = [_matrix(r, int(1000 * 100 ** u)) for u in r.random(48)]
    fmts = ["sell", "sell_sorted", "sell_c_s", "csr_naive"] * 12

    def least():
        best = float("inf")
        for _ in range(5):
            t = time.perf_counter()
            b = sb.Batch(mats, fmts)
            best = min(best, time.perf_counter() - t)
            del b
        return best

    alone = least()
    alive = [sb.Batch(mats, fmts) for _ in range(4)]
    beside = least()
    assert len(alive) == 4 and beside < 2 * alone, (alone, beside)


def _device_matrix(torch, entries, m=100000):
    """Rows of equal length on the GPU: 12 bytes an entry, arrays of less than 128 MB each."""
    k = entries // m
    rp = torch.arange(m + 1, dtype=torch.int32, device="cuda") * k
    ci = torch.arange(k, dtype=torch.int32, device="cuda").repeat(m)
    return rp, ci, torch.ones(k * m, dtype=torch.float64, device="cuda")


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_unused_memory_is_kept_beside_many_matrices(sb):
    """Matrices that hold more than a pool keeps do not make it give back what is free."""
    import torch

    big, small = _device_matrix(torch, 10_000_000), _device_matrix(torch, 1_000_000)
    held = [sb.csr_to_format(*big, format="csr_naive", kernel=4) for _ in range(7)]      # 840 MB of arrays
    other = sb.csr_to_format(*big, format="csr_naive", kernel=4)
    before = _free(torch)
    other.destroy()
    for _ in range(3):                                   # conversions synchronise
        sb.csr_to_format(*small, format="csr_naive").destroy()
    assert _free(torch) - before < 32 * MB               # the 120 MB of `other` wait for the next conversion
    for h in held:
        h.destroy()
    for _ in range(3):
        sb.csr_to_format(*small, format="csr_naive").destroy()
    assert _free(torch) - before >= 840 * MB + 120 * MB - KEEP - 64 * MB


class _OnlyFree:
    """Leaves `left` bytes of the device free while it lives."""

    def __init__(self, torch, left):
        self.torch, self.left = torch, left

    def __enter__(self):
        self.torch.cuda.empty_cache()
        self.fill = self.torch.empty(_free(self.torch) - self.left, dtype=self.torch.uint8, device="cuda")

    def __exit__(self, *exc):
        del self.fill
        self.torch.cuda.empty_cache()


def test_a_large_array_takes_what_the_pools_keep(sb):
    """200 MB free and more kept in the pool: a 240 MB array of values still finds its place."""
    import torch

    csr = _device_matrix(torch, 30_000_000)
    expect = sb.csr_to_format(*csr, format="csr_naive", kernel=4).spmv(torch.ones(100000, dtype=torch.float64, device="cuda"))
    x = torch.ones(100000, dtype=torch.float64, device="cuda")
    y = torch.empty_like(expect)
    kept = [sb.csr_to_format(*_device_matrix(torch, 10_000_000), format="csr_naive", kernel=4) for _ in range(4)]
    for h in kept:                                       # 480 MB stay in the pool
        h.destroy()
    with _OnlyFree(torch, 200 * MB):
        h = sb.csr_to_format(*csr, format="csr_naive", kernel=4)
        h.spmv(x, y)
        h.destroy()
    assert torch.equal(y, expect)

def test_an_allocation_without_memory_leaves_captures_alone(sb):
    """Conversions of another thread until the device is full: refused, and the capture goes on."""
    import torch

    csr = _device_matrix(torch, 10_000_000)
    x = torch.ones(100000, dtype=torch.float64, device="cuda")
    held, status = [], []
    mf = sb.csr_to_format(*csr, format="csr_naive", kernel=4)
    expect, y = mf.spmv(x), torch.zeros_like(x)

    def convert():
        try:
            while len(held) < 20:
                held.append(sb.csr_to_format(*csr, format="csr_naive", kernel=4))
        except sb.SpmvError as e:
            status.append(e.status)

    with _OnlyFree(torch, 200 * MB):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, capture_error_mode="thread_local"):
            mf.spmv(x, y)
            t = threading.Thread(target=convert)
            t.start()
            t.join()
            mf.spmv(x, y)
        g.replay()
        torch.cuda.synchronize()
        for h in held:
            h.destroy()
    assert status == [sb._capi.SPMV_ERR_NOMEM]
    assert torch.equal(y, expect)


def test_release_memory(sb):
    import torch

    csr = _device_matrix(torch, 10_000_000)
    sb.release_memory()
    before = _free(torch)
    held = [sb.csr_to_format(*csr, format="csr_naive", kernel=4) for _ in range(3)]
    for h in held:
        h.destroy()
    assert before - _free(torch) >= 300 * MB             # kept for the next conversions
    sb.release_memory()
    assert before - _free(torch) < 32 * MB


def test_a_refused_conversion_leaves_no_error_behind(sb):
    """After a conversion without memory the next launches, the library's and torch's, find no error."""
    import torch

    csr = _device_matrix(torch, 10_000_000)
    x = torch.ones(100000, dtype=torch.float64, device="cuda")
    h = sb.csr_to_format(*csr, format="csr_naive", kernel=0)
    expect, y = h.spmv(x), torch.zeros_like(x)
    sb.release_memory()
    with _OnlyFree(torch, 60 * MB):
        with pytest.raises(sb.SpmvError) as refused:
            sb.csr_to_format(*csr, format="csr_naive", kernel=0)
        assert refused.value.status == sb._capi.SPMV_ERR_NOMEM
        h.spmv(x, y)
        z = y + 0.0
    assert torch.equal(z, expect)
