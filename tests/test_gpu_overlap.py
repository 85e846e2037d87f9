"""Launches that overlap their predecessors: an SpMV may start before the kernel that writes its
x has ended, so chains of dependent kernels, enqueued without waiting, give what the same chain
gives with a wait after every step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [("csr_naive", 3000, {}), ("csr_naive", 200000, {}), ("csr_vec", 3000, dict(vec_len=4)),
         ("csr_vec", 200000, dict(vec_len=4)), ("sell_sorted", 200000, dict(vec_len=4)), ("sell_c_s", 3000, {}),
         ("sell_c_s", 200000, {}), ("csr_naive", 200000, dict(value_type="f32")), ("csr_naive", 3000, dict(value_type="f32"))]


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("fmt,m,kw", FORMS)
def test_dependent_chain(sb, fmt, m, kw, captured):
    import torch

    r = np.random.default_rng(m)
    lengths = r.integers(10, 31, m)
    rp = np.zeros(m + 1, np.int32)
    np.cumsum(lengths, out=rp[1:])
    start = r.integers(0, m - 32, m)
    ci = (np.repeat(start, lengths) + np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)).astype(np.int32)
    v = r.uniform(-1, 1, rp[-1]) / 8
    mf = sb.csr_to_format(rp, ci, v, format=fmt, **kw)
    x0 = torch.from_numpy(r.uniform(-1, 1, m)).cuda()
    if kw.get("value_type") == "f32":
        x0 = x0.float()

    def chain(x, y, z, wait):
        def done():
            if wait:
                torch.cuda.synchronize()

        for k in range(12):
            mf.spmv(x, y)                    # SpMV after SpMV: y is the next one's x
            done()
            mf.spmv(y, z)
            done()
            torch.mul(z, 0.5, out=x)         # a kernel that writes x, then the SpMV that reads it
            x.add_(0.25)
            done()
        return x

    ref = chain(x0.clone(), torch.empty_like(x0), torch.empty_like(x0), True)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    x, y, z = x0.clone(), torch.empty_like(x0), torch.empty_like(x0)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for _ in range(5):
            if captured:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s):
                    x.copy_(x0)
                    chain(x, y, z, False)
                g.replay()
            else:
                x.copy_(x0)
                chain(x, y, z, False)
            s.synchronize()
            assert torch.equal(x, ref)
