"""Conversions, SpMVs and destruction from several threads and streams at once: the pools that
their memory comes from hand a block on only when the work on it is done."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_share_the_pools(sb, orc):
    import torch

    cases = []
    for k, (fmt, kw) in enumerate([("csr_naive", {}), ("sell_c_s", {}), ("sell", dict(vec_len=4)), ("csr_vec", dict(vec_len=4))]):
        m = 20000 + 997 * k
        r = np.random.default_rng(k)
        lengths = r.integers(0, 30, m)
        rp = np.zeros(m + 1, np.int32)
        np.cumsum(lengths, out=rp[1:])
        ci = (np.repeat(r.integers(0, m - 64, m), lengths) + np.arange(rp[-1]) - np.repeat(rp[:-1], lengths)).astype(np.int32)
        v, x = r.uniform(-1, 1, rp[-1]), r.uniform(-1, 1, m)
        ref = {"csr_naive": lambda: orc.csr_spmv(rp, ci, v, x),
               "csr_vec": lambda: orc.csr_vec_spmv(rp, ci, v, x, 4),
               "sell": lambda: orc.sell_spmv(orc.sell_convert(rp, ci, v, 4, 8), m, 4, x),
               "sell_c_s": lambda: orc.sellcs_spmv(orc.sellcs_convert(rp, ci, v, 32, 512), m, 32, x)}[fmt]()
        cases.append((fmt, kw, rp, ci, v, x, ref))
    wrong = []

    def work(fmt, kw, rp, ci, v, x, ref):
        stream = torch.cuda.Stream()
        xd = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        for _ in range(12):
            mf = sb.csr_to_format(rp, ci, v, format=fmt, **kw)
            with torch.cuda.stream(stream):
                y = mf.spmv(xd)
            mf.destroy()                                  # before the SpMV is waited for
            stream.synchronize()
            if not np.array_equal(y.cpu().numpy().view(np.uint64), ref.view(np.uint64)):
                wrong.append(fmt)

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
