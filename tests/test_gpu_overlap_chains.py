"""Overlapped launches in chains of nothing but SpMVs: buffers read, written and read again by turns
(an iteration's a -> b, b -> a), and SpMVs behind a join of two streams.  Entries and vectors are
whole numbers small enough for every sum to be exact, so the chains with a wait after each step
give the same bits in every format (FP32 rows have one order in any case)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 12               # at most 6 entries of up to 3 a row: 18^12 < 2^53

FORMS = [("csr_naive", 3000, {}), ("csr_naive", 200000, {}), ("csr_naive", 1000000, {}), ("csr_vec", 1000000, dict(vec_len=4)),
         ("sell", 1000000, dict(vec_len=4)), ("sell_c_s", 3000, {}), ("sell_c_s", 200000, {}), ("sell_c_s", 3000, dict(sellcs_c=64)),
         ("div_rf", 3000, {}), ("div_rf", 200000, {}), ("div_rf", 200000, dict(vec_len=32, div_packet_vals=64)),
         ("div_rf", 1000000, dict(vec_len=8, div_packet_vals=1024)),
         ("csr_naive", 3000, dict(value_type="f32")), ("csr_naive", 1500000, dict(value_type="f32"))]


def _matrix(m, r):
    lengths = r.integers(0, 7, m)
    rp = np.zeros(m + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    ci = (np.repeat(r.integers(0, m - 6, m), lengths) + np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)).astype(np.int32)
    return rp, ci, r.integers(-3, 4, rp[-1]).astype(np.float64)


def _compare(torch, chain, x0, captured):
    """`chain(wait)` from x0: in order without waits, eager or captured, against waits everywhere."""
    ref = chain(torch.cuda.synchronize)
    torch.cuda.synchronize()
    ref = [t.clone() for t in ref]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for _ in range(6):
            if captured:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s):
                    got = chain(lambda: None)
                g.replay()
            else:
                got = chain(lambda: None)
            s.synchronize()
            for a, b in zip(got, ref):
                assert torch.equal(a, b)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("fmt,m,kw", FORMS)
def test_by_turns(sb, fmt, m, kw, captured):
    import torch

    r = np.random.default_rng(m)
    mf = sb.csr_to_format(*_matrix(m, r), format=fmt, **kw)
    x0 = torch.from_numpy(r.integers(-1, 2, m).astype(np.float32 if "value_type" in kw else np.float64)).cuda()
    a, b = torch.empty_like(x0), torch.empty_like(x0)

    def chain(wait):
        a.copy_(x0)
        for _ in range(STEPS // 2):
            mf.spmv(a, b)
            wait()
            mf.spmv(b, a)
            wait()
        return a, b

    _compare(torch, chain, x0, captured)


@pytest.mark.parametrize("graph", [False, True])
def test_batches_by_turns(sb, graph):
    import torch

    r = np.random.default_rng(7)
    mats = [(*_matrix(m, r), m, m) for m in (3000, 40000, 1025, 90000, 300, 64, 20000, 7000)]
    batch = sb.Batch(mats, ["sell", "sell_sorted", "sell_c_s", "csr_naive"] * 2)
    x0 = torch.from_numpy(r.integers(-1, 2, batch.total_x).astype(np.float64)).cuda()
    a, b = torch.empty_like(x0), torch.empty_like(x0)

    def chain(wait):
        a.copy_(x0)
        for _ in range(STEPS // 2):
            batch.spmv(a, b, graph=graph)
            wait()
            batch.spmv(b, a, graph=graph)
            wait()
        return a, b

    _compare(torch, chain, x0, False)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("fmt,m,kw", [FORMS[0], FORMS[2], FORMS[6], FORMS[9]])
def test_behind_a_join(sb, fmt, m, kw, captured):
    """b on one stream, c from it on another, d beside that, then SpMVs of c and of d behind the join."""
    import torch

    r = np.random.default_rng(m + 1)
    mf = sb.csr_to_format(*_matrix(m, r), format=fmt, **kw)
    x0 = torch.from_numpy(r.integers(-1, 2, m).astype(np.float64)).cuda()
    a, b, c, d, e = (torch.empty_like(x0) for _ in range(5))
    side = torch.cuda.Stream()

    def chain(wait):
        main = torch.cuda.current_stream()
        a.copy_(x0)
        for _ in range(STEPS // 4):
            mf.spmv(a, b)
            wait()
            side.wait_stream(main)
            with torch.cuda.stream(side):
                mf.spmv(b, c)
            wait()
            mf.spmv(b, d)
            wait()
            main.wait_stream(side)
            mf.spmv(c, e)
            wait()
            mf.spmv(d, a)
            wait()
        return a, b, c, d, e

    _compare(torch, chain, x0, captured)
