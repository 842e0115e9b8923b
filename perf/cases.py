"""Performance cases of the compressed matrix products, as a program that uses this package calls them.

Two kinds of caller exist and both are covered: the instruction layer, which hands over host arrays block by block and
goes through the ``CLALib*`` classes (``io`` = "host"), and iterative algorithms that keep the compressed block and
their vectors on the GPU and call the device-buffer entry points of the C ABI on the current stream (``io`` = "dev").

A case is a flat dict:

* ``op``    "xv" X %*% V, "ytx" Yt %*% X, "chain" t(X) %*% (w * (X %*% v)), "tsmm" t(X) %*% X, "decompress"
* ``kind``  "bytes" single-column dense-map groups of up to 256 tuples, "chars" the same with more (16-bit maps, skewed
            ids), "mixed" 40 % dense-map columns of 4 tuples / 30 % columns with 5 % listed rows (sparse default) / 20 %
            run-length columns / 10 % uncompressed columns
* ``rows``, ``cols``; ``card`` tuples per dictionary (0: every column its own, uniform in 2..255); ``k`` columns of V
  or rows of Yt; ``weighted`` whether the chain carries w.
"""
import math

import numpy as np
import torch

from systemds_b200 import (CHAIN_XtXv, CHAIN_XtwXv, CLALibDecompress, CLALibLeftMultBy, CLALibMMChain, CLALibRightMultBy,
                           CLALibTSMM, CompressedMatrixBlock, native)
from systemds_b200.colgroup import ColGroupDDC, ColGroupRLE, ColGroupSDCZeros, ColGroupUncompressedDev
from systemds_b200.mapping import MAP_BIT, DeviceMap, MapToFactory
from systemds_b200.offset import OffsetFactory


def _case(name, op, kind, rows, cols, card=0, k=1, io="dev", weighted=False):
    c = {"op": op, "kind": kind, "rows": rows, "cols": cols, "card": card, "k": k, "io": io, "weighted": weighted}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one 1000-row block of a blocked matrix, host arrays in and out: what a distributed X %*% v does per block
        _case("block_xv", "xv", "bytes", 1_000, 100, io="host"),
        # conjugate-gradient step on a small training set that fits the L2 cache: launches and latency count
        _case("chain_small", "chain", "bytes", 50_000, 100),
        # scoring a million rows with a linear model, 16-value dictionaries (ids of binned features)
        _case("xv_1m", "xv", "bytes", 1_000_000, 100, card=16),
        # gradient t(y) %*% X over ten million rows, full byte dictionaries: the headline workload
        _case("ytx_10m", "ytx", "bytes", 10_000_000, 200, card=256),
        # linear-regression conjugate gradient over a tall and wide shard, cardinality 2..255
        _case("lmcg_6m", "chain", "bytes", 6_250_000, 1_000),
        # iteratively reweighted least squares on a real-life mix of encodings, ragged row count
        _case("chain_mixed", "chain", "mixed", 999_983, 500, weighted=True),
        # multi-class scoring / projection on the mix of encodings, 64 result columns
        _case("xV_mixed", "xv", "mixed", 1_000_000, 500, k=64),
        # class-probability gradients: eight left rows against the mix of encodings
        _case("ytX_mixed", "ytx", "mixed", 500_000, 250, k=8),
        # direct-solve normal equations, 1000-value dictionaries with skewed ids
        _case("tsmm_chars", "tsmm", "chars", 4_000_000, 100, card=1_000),
        # normal equations / covariance on the mix of encodings, more columns than one result tile
        _case("tsmm_mixed", "tsmm", "mixed", 200_000, 250),
        # projection of byte-coded columns on ten components
        _case("xV_bytes", "xv", "bytes", 1_000_000, 200, card=256, k=10),
        # decompress for an operator that has no compressed form
        _case("decompress_mixed", "decompress", "mixed", 250_001, 500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: sizes log-uniform and mostly odd, never more work than the largest listed case of
    its operation."""
    op = rng.choice(["xv", "xv", "ytx", "ytx", "chain", "chain", "tsmm", "decompress"])
    kind = rng.choice(["bytes", "bytes", "mixed", "mixed", "chars"])
    cols = _log(rng, 20, 1000) if kind == "bytes" and op != "tsmm" else _log(rng, 30, 500 if op != "tsmm" else 250)
    card = 0 if kind == "mixed" else (rng.randint(300, 2000) if kind == "chars" else rng.choice([0, 0, 4, 16, 100, 256]))
    k = 1
    if op == "xv" and rng.random() < 0.5:
        k = _log(rng, 2, 64)
    if op == "ytx" and rng.random() < 0.5:
        k = _log(rng, 2, 8)
    # cells of the matrix, from one block to the largest listed matrix of the kind
    most = 2.0e9 if kind == "bytes" else (5.0e8 if kind == "mixed" else 4.0e8)
    if op == "tsmm":
        most = min(most, 4.0e10 / cols)
    if op == "decompress":
        most = 1.25e8
    if op == "xv" and k > 1:
        most = min(most, 3.2e10 / k / (1 if kind != "chars" else 4))
    if op == "ytx" and k > 1:
        most = min(most, 1.0e9 / k)
    rows = max(500, _log(rng, 1.0e5, most) // cols)
    io = "host" if rows <= 20_000 and op != "decompress" and rng.random() < 0.5 else "dev"
    return _case(None, op, kind, rows, cols, card, k, io, op == "chain" and rng.random() < 0.5)


# ---- inputs -------------------------------------------------------------------------------------------------------
def _byte_map(n, card, gen):
    t = MapToFactory.type_for(n, card)
    if t == MAP_BIT:  # long[] words, one bit per row
        w = torch.randint(0, 256, ((n + 63) // 64 * 8,), dtype=torch.uint8, device="cuda", generator=gen)
        w[(n + 7) // 8:] = 0
        if n % 8:
            w[n // 8] &= (1 << (n % 8)) - 1
        return DeviceMap(t, n, card, w.data_ptr(), w.numel(), owner=w)
    ids = torch.randint(0, card, (n,), dtype=torch.uint8, device="cuda", generator=gen)
    return DeviceMap(t, n, card, ids.data_ptr(), n, owner=ids)


def _char_map(n, card, cdf, gen):
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    ids = torch.searchsorted(cdf, u).clamp_(max=card - 1).to(torch.int16)
    return DeviceMap(MapToFactory.type_for(n, card), n, card, ids.data_ptr(), n * 2, owner=ids)


def _mixed_counts(cols):
    ddc, sdc, rle = int(cols * 0.4), int(cols * 0.3), int(cols * 0.2)
    return ddc, sdc, rle, cols - ddc - sdc - rle


def _matrix(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 1_000_003 + 17)
    rng = np.random.Generator(np.random.Philox(key=seed))
    n, cols, groups = c["rows"], c["cols"], []
    if c["kind"] == "bytes":
        cards = rng.integers(2, 256, size=cols) if c["card"] == 0 else np.full(cols, c["card"])
        for j in range(cols):
            groups.append(ColGroupDDC([j], rng.standard_normal((cards[j], 1)), _byte_map(n, int(cards[j]), gen)))
    elif c["kind"] == "chars":
        w = 1.0 / np.power(np.arange(1, c["card"] + 1, dtype=np.float64), 1.1)
        cdf = torch.from_numpy(np.cumsum(w / w.sum())).cuda()
        for j in range(cols):
            groups.append(ColGroupDDC([j], rng.uniform(-1.0, 1.0, (c["card"], 1)), _char_map(n, c["card"], cdf, gen)))
    else:
        ddc, sdc, rle, unc = _mixed_counts(cols)
        for j in range(ddc):
            groups.append(ColGroupDDC([j], rng.standard_normal((4, 1)), _byte_map(n, 4, gen)))
        for j in range(ddc, ddc + sdc):  # 5 % of the rows listed
            rows = torch.nonzero(torch.rand(n, device="cuda", generator=gen) < 0.05).reshape(-1).cpu().numpy()
            ids = rng.integers(0, 8, size=rows.shape[0])
            groups.append(ColGroupSDCZeros([j], n, rng.standard_normal((8, 1)), OffsetFactory.createOffset(rows),
                                           MapToFactory.create_from(ids, 8)))
        for j in range(ddc + sdc, ddc + sdc + rle):  # geometric runs of mean 1000, neighbouring runs differ
            lens = rng.geometric(1.0e-3, size=int(n / 1000 * 1.5) + 64)
            ends = np.minimum(np.cumsum(lens), n)
            starts = np.concatenate([[0], ends[:-1]])
            keep = ends > starts
            starts, ends = starts[keep], ends[keep]
            ends[-1] = n
            vals = np.cumsum(rng.integers(1, 32, size=starts.shape[0])) % 32
            groups.append(ColGroupRLE.from_runs([j], rng.standard_normal((32, 1)), starts, ends - starts, vals, n))
        dense = torch.randn((n, unc), dtype=torch.float64, device="cuda", generator=gen)
        groups.append(ColGroupUncompressedDev(list(range(cols - unc, cols)), n, dense.data_ptr(), owner=dense))
    torch.cuda.synchronize()  # the block is built on a stream of its own
    x = CompressedMatrixBlock(n, cols, groups).to_device(torch.cuda.current_device())
    x._colGroups = []  # the block keeps its own copy: drop the generator's
    return x, gen, rng


def prepare(case, seed):
    x, gen, rng = _matrix(case, seed)
    n, cols, k, op = case["rows"], case["cols"], case["k"], case["op"]
    s = {"case": case, "x": x}

    def normal(*shape):
        if case["io"] == "host":
            return rng.standard_normal(shape)
        return torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)

    def result(*shape):
        if case["io"] == "dev":
            s["out"] = torch.empty(shape, dtype=torch.float64, device="cuda")

    if op == "xv":
        s["v"] = normal(cols, k)
        result(n, k)
    elif op == "ytx":
        s["y"] = normal(k, n)
        result(k, cols)
    elif op == "chain":
        s["v"] = normal(cols)
        s["w"] = None
        if case["weighted"]:
            z = normal(n)
            s["w"] = 1.0 / (2.0 + np.exp(z) + np.exp(-z)) if case["io"] == "host" else torch.sigmoid(z) * torch.sigmoid(-z)
        result(cols)
    elif op == "tsmm":
        result(cols, cols)
    else:
        result(n, cols)
    return s


# ---- the calls ----------------------------------------------------------------------------------------------------
def run(state):
    c, x = state["case"], state["x"]
    op = c["op"]
    if c["io"] == "host":
        if op == "xv":
            return CLALibRightMultBy.rightMultByMatrix(x, state["v"])
        if op == "ytx":
            return CLALibLeftMultBy.leftMultByMatrix(x, state["y"])
        if op == "chain":
            return CLALibMMChain.mmChain(x, state["v"], state["w"], CHAIN_XtXv if state["w"] is None else CHAIN_XtwXv)
        if op == "tsmm":
            return CLALibTSMM.leftMultByTransposeSelf(x)
        return CLALibDecompress.decompress(x)
    lib, h, out = native.lib(), x.handle(), state["out"]
    stream = torch.cuda.current_stream().cuda_stream
    if op == "xv":
        rc = lib.cla_rmm_dev(h, state["v"].data_ptr(), c["cols"], c["k"], out.data_ptr(), stream)
    elif op == "ytx":
        rc = lib.cla_lmm_dev(h, state["y"].data_ptr(), c["k"], out.data_ptr(), stream)
    elif op == "chain":
        w = state["w"]
        rc = lib.cla_mmchain_dev(h, state["v"].data_ptr(), 0 if w is None else w.data_ptr(),
                                 CHAIN_XtXv if w is None else CHAIN_XtwXv, out.data_ptr(), 0, stream)
    elif op == "tsmm":
        rc = lib.cla_tsmm_dev(h, out.data_ptr(), stream)
    else:
        rc = lib.cla_decompress_dev(h, out.data_ptr(), stream)
    native.check(rc)
    return out


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def work(case):
    n, cols, k, op = case["rows"], case["cols"], case["k"], case["op"]
    if case["kind"] == "mixed":
        ddc, sdc, rle, unc = _mixed_counts(cols)
        index = n * (ddc + sdc * 0.05 * 2 + rle * 4.0e-3 + unc * 8) + 8.0 * (4 * ddc + 8 * sdc + 32 * rle)
        terms = n * (ddc + sdc * 0.05 + rle * 2.0e-3 + unc * 2)  # adds per result column (a product more where dense)
    else:
        card = case["card"] or 128
        index = n * cols * (2 if case["kind"] == "chars" else 1) + 8.0 * card * cols
        terms = n * cols
    if op == "xv":
        return {"bytes": index + 8.0 * k * (n + cols), "flops": terms * k}
    if op == "ytx":
        return {"bytes": index + 8.0 * k * (n + cols), "flops": terms * k}
    if op == "chain":  # both directions need the whole matrix, and the vector between them does not fit on chip
        return {"bytes": index + 16.0 * cols + (8.0 * n if case["weighted"] else 0.0), "flops": 2.0 * terms}
    if op == "tsmm":
        return {"bytes": index + 8.0 * cols * cols, "flops": 1.0 * n * cols * (cols + 1)}
    return {"bytes": index + 8.0 * n * cols, "flops": 1.0 * n * cols}


def tolerance(case):
    """Double precision throughout: sums of up to a thousand terms along a row, of up to ten million along a column."""
    if case["op"] == "decompress":
        return "exact"  # the dictionary values themselves
    return {"rel": 1.0e-13 if case["op"] == "xv" else 1.0e-12}
