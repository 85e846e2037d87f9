"""Destroying a matrix waits for the SpMVs that still use it, on whatever stream, before its memory
can be handed on -- also while a stream is being captured -- and leaves the capture intact."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = 40000
SLEEP = 100_000_000      # cycles: about 50 ms at 1,965 MHz


def _matrix(sb, seed, **kw):
    r = np.random.default_rng(seed)
    lengths = r.integers(0, 30, M)
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    ci = (np.repeat(r.integers(0, M - 64, M), lengths) + np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)).astype(np.int32)
    return sb.csr_to_format(rp, ci, r.uniform(-1, 1, rp[-1]), format="csr_naive", **kw)


def _destroy_behind_work(torch, mf, x, y, side):
    """An SpMV behind 50 ms of work on `side`, then destroy(): was the work over when it returned?"""
    done = torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)
        mf.spmv(x, y)
        done.record(side)
    assert not done.query()
    mf.destroy()
    return done.query()


def test_destroy_waits_for_other_streams(sb):
    import torch

    x = torch.rand(M, dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    side = torch.cuda.Stream()
    mf = _matrix(sb, 1)
    expect = mf.spmv(x)
    torch.cuda.synchronize()
    assert _destroy_behind_work(torch, mf, x, y, side)
    assert torch.equal(y, expect)


@pytest.mark.parametrize("same_thread", [False, True])
def test_destroy_during_a_capture(sb, same_thread):
    """In a capture of the calling thread (global mode, torch's default) and in one of another
    thread: the destroyed matrix's SpMV is over, the capture goes on and replays."""
    import torch

    x = torch.rand(M, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    z = torch.zeros_like(x)
    kept, gone = _matrix(sb, 2), _matrix(sb, 3)
    expect, gone_expect = kept.spmv(x), gone.spmv(x)
    side, over, gone_event = torch.cuda.Stream(), [], torch.cuda.Event()
    torch.cuda.synchronize()
    if same_thread:                                      # enqueued before: a capture allows no query of it
        with torch.cuda.stream(side):
            torch.cuda._sleep(SLEEP)
            gone.spmv(x, z)
            gone_event.record(side)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global" if same_thread else "thread_local"):
        kept.spmv(x, y)
        if same_thread:
            gone.destroy()
        else:
            t = threading.Thread(target=lambda: over.append(_destroy_behind_work(torch, gone, x, z, side)))
            t.start()
            t.join()
        kept.spmv(x, y)
    assert gone_event.query() if same_thread else over == [True]
    assert torch.equal(z, gone_expect)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, expect)
    after = _matrix(sb, 2)
    assert torch.equal(after.spmv(x), expect)
