"""Performance cases: the SpMV calls of this package over the range of matrices it is used on.

A case names a matrix by the parameters of its structure, the storage format with its options
and how the call is made:

    call "device"   the solver's inner step: a converted matrix, x and y on the GPU
    call "host"     the drop-in's step: Matrix_Format::spmv with host x and y
    call "convert"  a new matrix: csr_to_format of host CSR arrays, then its first host SpMV
    call "batch"    many uneven matrices in one captured launch

The matrices are made with torch on the GPU (integer arithmetic after the random draws, so a seed
always names the same matrix): row lengths normal or gamma, a geometric tail of `skew` times longer
rows at the top, columns in a window of `bw` of the width around the diagonal or the middle, broken
into runs (`neigh`: average neighbours of an entry, 2 = one run a row) and shared by pairs of rows
(`cross`).  These are the parameters of the reference's artificial matrix generator.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def package():
    if "spmv_dare_b200" in sys.modules:
        return sys.modules["spmv_dare_b200"]
    pkg = os.path.join(ROOT, "spmv-dare_b200")
    spec = importlib.util.spec_from_file_location("spmv_dare_b200", os.path.join(pkg, "__init__.py"),
                                                  submodule_search_locations=[pkg])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["spmv_dare_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# The two single-matrix configurations of the benchmark, by the structure of the matrices.
NORMAL_100K = dict(rows=100000, cols=100000, avg=10.0, std=2.0, dist="normal", skew=0.0, bw=0.3, place="middle",
                   neigh=1.0, cross=0.5, values="uniform")
GAMMA_4M = dict(rows=4000000, cols=4000000, avg=20.0, std=0.5, dist="gamma", skew=100.0, bw=0.15, place="middle",
                neigh=1.9, cross=0.3, values="uniform")


def listed():
    return [
        # the smallest systems (coarse multigrid levels, the smoke matrix): launch latency counts
        dict(name="csr_naive_2k", call="device", format="csr_naive", rows=2000, cols=2000, avg=20.0, std=15.0,
             dist="gamma", skew=20.0, bw=0.3, place="middle", neigh=1.5, cross=0.3, values="uniform"),
        # the benchmark's small configuration: fits in L2, scattered columns
        dict(name="csr_naive_100k", call="device", format="csr_naive", **NORMAL_100K),
        # the headline: the 4M-row matrix in CSR
        dict(name="csr_naive_4m", call="device", format="csr_naive", **GAMMA_4M),
        # a mid-size matrix with uneven rows and an odd row count, four-lane CSR
        dict(name="csr_vec_1m", call="device", format="csr_vec", rows=1000003, cols=1000003, avg=33.0, std=14.0,
             dist="gamma", skew=30.0, bw=0.1, place="diagonal", neigh=1.5, cross=0.4, values="uniform"),
        # SELL with the reference's slices of 4 rows, rows of similar length (meshes)
        dict(name="sell_2m", call="device", format="sell", rows=2000000, cols=2000000, avg=26.0, std=3.0,
             dist="normal", skew=0.0, bw=0.05, place="diagonal", neigh=1.6, cross=0.5, values="uniform"),
        # SELL over sorted rows: irregular lengths, an odd, rectangular shape
        dict(name="sell_sorted_700k", call="device", format="sell_sorted", rows=700001, cols=900007, avg=30.0,
             std=18.0, dist="gamma", skew=60.0, bw=0.3, place="middle", neigh=1.2, cross=0.4, values="uniform"),
        # the 4M-row matrix in SELL-C-sigma (C = 32, sigma = 512)
        dict(name="sell_c_s_4m", call="device", format="sell_c_s", **GAMMA_4M),
        # compressed values and indices, the reference's defaults (4 lanes, 16,384-value packets)
        dict(name="div_rf_1m", call="device", format="div_rf",
             **dict(GAMMA_4M, rows=1000001, cols=1000001)),
        # few distinct values (stencils, repeated elements), as many lanes as a warp
        dict(name="div_rf_few_300k", call="device", format="div_rf", rows=300007, cols=300007, avg=27.0, std=4.0,
             dist="normal", skew=0.0, bw=0.05, place="diagonal", neigh=1.6, cross=0.5, values="few", vec_len=32,
             div_packet_vals=4096),
        # FP32 storage with compensated rows on the 4M-row matrix
        dict(name="f32_4m", call="device", format="csr_naive", value_type="f32", **GAMMA_4M),
        # a batch of uneven matrices in the four batchable formats, one graph replay
        dict(name="batch_mixed_48", call="batch", format="mixed", count=48, rows_lo=1000, rows_hi=100000),
        # the reference's driver on a new matrix: conversion of host arrays and the first host SpMV
        dict(name="convert_sell_c_s_300k", call="convert", format="sell_c_s",
             **dict(GAMMA_4M, rows=300007, cols=300007, avg=28.0, std=12.0)),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choices(["device", "host", "convert", "batch"], [10, 1, 1, 1])[0]
    if call == "batch":
        lo = int(_log_uniform(rng, 1000, 4000))
        return dict(call="batch", format=rng.choice(["mixed", "csr_naive"]), count=rng.randint(8, 48), rows_lo=lo,
                    rows_hi=int(lo * _log_uniform(rng, 4, 25)))
    fmt = rng.choice(["csr_naive", "csr_naive", "csr_vec", "sell", "sell_sorted", "sell_c_s", "sell_c_s", "div_rf", "f32"])
    most = 20e6 if fmt == "div_rf" else 80e6        # entries, no more than the largest listed case of the kind
    if call != "device":
        most = 8e6
    avg = round(rng.uniform(5.0, 60.0), 2)
    rows = int(_log_uniform(rng, 1e3, min(4e6, most / avg)))
    case = dict(call=call, format="csr_naive" if fmt == "f32" else fmt, rows=rows,
                cols=rows if rng.random() < 0.8 else int(rows * rng.uniform(0.8, 1.5)), avg=avg,
                std=round(rng.uniform(0.02, 0.8) * avg, 2), dist=rng.choice(["normal", "gamma"]),
                skew=round(rng.choice([0.0, rng.uniform(0.0, 100.0)]), 1), bw=round(rng.uniform(0.02, 0.5), 3),
                place=rng.choice(["diagonal", "middle"]), neigh=round(rng.uniform(1.0, 1.95), 2),
                cross=round(rng.uniform(0.2, 0.5), 2), values="uniform")
    if fmt == "f32":
        case["value_type"] = "f32"
    elif fmt in ("csr_vec", "sell", "sell_sorted"):
        case["vec_len"] = rng.choice([4, 4, 4, 8])
    elif fmt == "sell_c_s":
        case["sellcs_c"], case["sellcs_sigma"] = rng.choice([(32, 512), (32, 256), (64, 1024)])
    elif fmt == "div_rf":
        case["vec_len"], case["div_packet_vals"] = rng.choice([(4, 16384), (4, 16384), (32, 4096), (32, 16384)])
        case["values"] = rng.choice(["uniform", "few"])
    return case


OPTIONS = ("vec_len", "sellcs_c", "sellcs_sigma", "div_packet_vals", "value_type")


def options(case):
    return {k: case[k] for k in OPTIONS if k in case}


# ------------------------------------------------------------------ matrices
def matrix(case, seed, dev="cuda"):
    """CSR tensors (int32 row_ptr, int32 ascending columns, float64 values), x: from the seed alone."""
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) * 7919 + 17)
    m, n, avg, std = case["rows"], case["cols"], case["avg"], case["std"]
    if case["dist"] == "normal":
        length = torch.randn(m, generator=g, device=dev, dtype=torch.float64) * std + avg
    else:
        # gamma of mean avg and deviation std: sum of exponentials of the nearest whole shape
        shape = max(1, round((avg / std) ** 2))
        if shape <= 16:
            length = torch.zeros(m, device=dev, dtype=torch.float64)
            for _ in range(shape):
                length -= torch.log(1.0 - torch.rand(m, generator=g, device=dev, dtype=torch.float64))
            length *= avg / shape
        else:                                       # close to normal
            length = torch.randn(m, generator=g, device=dev, dtype=torch.float64) * std + avg
    top = min(avg * (1.0 + case["skew"]), 0.4 * n)
    if case["skew"] > 0:                            # the long rows: about 1% of the entries
        tau = max(1.0, 0.01 * m * avg / top)
        length += top * torch.exp(-torch.arange(m, device=dev, dtype=torch.float64) / tau)
    length = length.round().long().clamp_(0, int(min(0.5 * n, top + 20 * avg)))
    # pairs of rows with the same columns
    src = torch.arange(m, device=dev)
    same = (torch.rand(m, generator=g, device=dev) < 2.0 * case["cross"]) & (src % 2 == 1)
    src = torch.where(same, src - 1, src)
    length = length[src]
    rp = torch.zeros(m + 1, dtype=torch.int64, device=dev)
    torch.cumsum(length, 0, out=rp[1:])
    nnz = int(rp[m])
    # whole-numbered gaps between a row's columns: none inside a run, exponential between runs
    row = torch.repeat_interleave(torch.arange(m, device=dev), length, output_size=nnz)
    k = torch.arange(nnz, device=dev) - rp[row]
    gap = (-256.0 * torch.log(1.0 - torch.rand(nnz, generator=g, device=dev))).long() + 1
    gap[(torch.rand(nnz, generator=g, device=dev) < 0.5 * case["neigh"]) & (k > 0)] = 0
    at = rp[src[row]] + k
    gap = gap[at]
    del at
    cum = torch.cumsum(gap, 0)
    first = torch.clamp(rp[:-1], max=max(nnz - 1, 0))
    base = (cum[first] - gap[first])[row] if nnz else cum
    cum -= base
    last = torch.clamp(rp[1:] - 1, min=0)
    end = (torch.rand(m, generator=g, device=dev) * 512.0).long()[src] + 1
    total = (cum[last] + end)[row] if nnz else cum  # the gap after the last column counts too
    window = torch.clamp(length * 2, min=int(case["bw"] * n)).clamp_(max=n)
    centre = (src * n) // max(m, 1) if case["place"] == "diagonal" else torch.full((m,), n // 2, device=dev)
    start = torch.minimum(torch.clamp(centre - window // 2, min=0), n - window)
    col = start[row] + k + ((window - length)[row] * cum) // total
    del gap, cum, base, total, k
    if case["values"] == "uniform":                 # k / 2^31, mapped to [-1, 1)
        v = torch.randint(0, 1 << 31, (nnz,), generator=g, device=dev).double() / (1 << 30) - 1.0
    else:                                           # some hundred values, as repeated elements give
        table = torch.rand(300, generator=g, device=dev, dtype=torch.float64) * 2.0 - 1.0
        v = table[(torch.rand(nnz, generator=g, device=dev, dtype=torch.float64) ** 2 * 300).long()]
    x = torch.rand(n, generator=g, device=dev, dtype=torch.float64) * 2.0 - 1.0
    return rp.int(), col.int(), v, x


def batch_cases(case):
    """The matrices of a batch, spread over the logarithm of the rows."""
    r = np.random.Generator(np.random.PCG64(case["count"]))
    out = []
    for i in range(case["count"]):
        rows = int(case["rows_lo"] * (case["rows_hi"] / case["rows_lo"]) ** r.uniform())
        avg = float(r.uniform(5.0, 60.0))
        out.append(dict(rows=rows, cols=rows, avg=avg, std=float(r.uniform(0.1, 0.8)) * avg,
                        dist="normal" if r.uniform() < 0.5 else "gamma", skew=float(r.uniform(0.0, 100.0)),
                        bw=float(r.uniform(0.01, 0.5)), place="middle", neigh=float(r.uniform(1.0, 1.95)),
                        cross=float(r.uniform(0.3, 0.5)), values="uniform"))
    return out


BATCH_FORMATS = ("sell", "sell_sorted", "sell_c_s", "csr_naive")


# ------------------------------------------------------------------ the measured calls
def prepare(case, seed):
    sb = package()
    if case["call"] == "batch":
        mats, xs, fmts = [], [], []
        for i, c in enumerate(batch_cases(case)):
            rp, ci, v, x = matrix(c, seed * 1000 + i)
            mats.append((rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy(), c["rows"], c["cols"]))
            xs.append(x)
            fmts.append(BATCH_FORMATS[i % 4] if case["format"] == "mixed" else case["format"])
        b = sb.Batch(mats, fmts)
        x = torch.cat(xs)
        return dict(case=case, batch=b, x=x, y=torch.zeros(b.total_y, dtype=torch.float64, device="cuda"))
    rp, ci, v, x = matrix(case, seed)
    if case["call"] == "convert":
        return dict(case=case, csr=(rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()), x=x.cpu().numpy(),
                    y=np.zeros(case["rows"]))
    mf = sb.csr_to_format(rp, ci, v, n=case["cols"], format=case["format"], **options(case))
    if case["call"] == "host":                      # pinned buffers, as the benchmark's driver keeps them
        f = torch.float64
        return dict(case=case, mf=mf, x=x.cpu().pin_memory().numpy(),
                    y=torch.zeros(case["rows"], dtype=f).pin_memory().numpy())
    if case.get("value_type") == "f32":
        x = x.float()
    return dict(case=case, mf=mf, x=x, y=torch.zeros(case["rows"], dtype=x.dtype, device="cuda"))


def run(state):
    case = state["case"]
    if case["call"] == "batch":
        return state["batch"].spmv(state["x"], state["y"], graph=True)
    if case["call"] == "convert":
        rp, ci, v = state["csr"]
        mf = package().csr_to_format(rp, ci, v, n=case["cols"], format=case["format"], **options(case))
        y = mf.spmv(state["x"], state["y"])
        mf.destroy()
        return y
    return state["mf"].spmv(state["x"], state["y"])


def _work_one(case):
    m, n, avg = case["rows"], case["cols"], case["avg"]
    nnz = m * avg * (1.01 if case["skew"] > 0 else 1.0)
    if case.get("value_type") == "f32":
        return nnz * 8 + 4 * (m + 1) + 4 * n + 4 * m, 2 * nnz
    per = 12.0
    if case["format"] == "div_rf":                  # coordinates, and where values differ a code and a payload
        per = 7.8 if case["values"] == "uniform" else 3.2
    return nnz * per + 4 * (m + 1) + 8 * n + 8 * m, 2 * nnz


def work(case):
    """The stored matrix and x read once, y written once."""
    if case["call"] == "batch":
        each = [_work_one(dict(c, format="csr_naive")) for c in batch_cases(case)]
    else:
        each = [_work_one(case)]
    return {"bytes": int(sum(e[0] for e in each)), "flops": int(sum(e[1] for e in each))}


def _exact_one(case, seed):
    rp, ci, v, x = matrix(case, seed)
    if case.get("value_type") == "f32":             # the variant's values and x, rounded once
        v, x = v.float().double(), x.float().double()
    prod = v * x[ci.long()]
    return torch.segment_reduce(prod, "sum", lengths=(rp[1:] - rp[:-1]).long(), initial=0.0)


def exact(case, seed):
    if case["call"] == "batch":
        return torch.cat([_exact_one(c, seed * 1000 + i) for i, c in enumerate(batch_cases(case))])
    y = _exact_one(case, seed)
    return y if case["call"] == "device" else y.cpu().numpy()
