"""The work that programs using this library have it do, as measurable cases.

A case is a dict of plain values naming a matrix family, its sizes, the value
types and the entry point. `listed()` gives the fixed cases, `draw(rng)` one
more case of the same ranges, `prepare(case, seed)` the inputs and handles a
program has in hand before the call, `run(state)` one pass through the public
entry points, `exact(case, seed)` the same result in 64 bits by plain torch.

Matrices are generated on the GPU from the seed alone. FP64 CSR handles are
created from device arrays, FP32 CSR and BSR handles from host arrays (the
entry points they have). Handles, kernel choices and batch schedules are made
in `prepare`: a program keeps them over many products with one matrix.
"""
import math
import random

import numpy as np
import torch

import perf_libs_sparse_b200 as pls

DEV = "cuda"
ZIPF_MAX = 4096
ZIPF_SHIFT = 1.8618  # P(len) ~ (len + q)^-2 on [1, 4096] with mean 16
ZIPF_MEAN = 16.0


# ------------------------------------------------------------------ cases

def listed():
    return [
        # A small operator inside an iterative solver: one product is a few
        # microseconds, so the call itself counts.
        {"name": "laplace-100-f64", "op": "spmv", "matrix": "laplace2d", "g": 100, "dtype": "f64",
         "storage": "native", "optimize": False, "trans": False, "alpha": 1.0, "beta": 0.0},
        # The plain CSR product of a handle that was never optimized, on a
        # 5-point Laplacian (the repository's first benchmark configuration).
        {"name": "laplace-512-f64", "op": "spmv", "matrix": "laplace2d", "g": 512, "dtype": "f64",
         "storage": "native", "optimize": False, "trans": False, "alpha": 1.0, "beta": 0.0},
        # Power-law rows with random columns (graphs), tuned by optimize: the
        # benchmark's headline product, and the largest one here.
        {"name": "powerlaw-4m-f64", "op": "spmv", "matrix": "zipf", "n": 4194304, "dtype": "f64",
         "storage": "native", "optimize": True, "trans": False, "alpha": 1.0, "beta": 0.0},
        # The same family with values held in FP32 (the opt-in storage mode)
        # and y updated in place, at a ragged size.
        {"name": "powerlaw-1m-f32store", "op": "spmv", "matrix": "zipf", "n": 1000003, "dtype": "f64",
         "storage": "fp32", "optimize": True, "trans": False, "alpha": 1.5, "beta": 0.5},
        # y = A^T x on a rectangular matrix (least squares, adjoint products),
        # optimized for the transposed operation.
        {"name": "rect-700k-trans-f64", "op": "spmv", "matrix": "uniform", "n": 700001, "ncols": 500009,
         "mean": 12, "dtype": "f64", "storage": "native", "optimize": True, "trans": True,
         "alpha": 1.0, "beta": 0.5},
        # Block matrices of coupled unknowns (8 per node): BSR product.
        {"name": "bsr8-spmv-f64", "op": "bsr_spmv", "mb": 60011, "per_row": 8, "bs": 8, "rowmajor": True,
         "dtype": "f64", "storage": "native", "alpha": 1.0, "beta": 0.0},
        # A 3-D stencil operator applied to a block of vectors (block Krylov
        # methods): the benchmark's SpMM configuration.
        {"name": "stencil-128-k32-f64", "op": "spmm", "matrix": "stencil27", "g": 128, "k": 32,
         "dtype": "f64", "storage": "native", "alpha": 1.0, "beta": 0.0},
        # The same operator with BF16 values and FP32 vectors, many vectors, a
        # grid that is no power of two.
        {"name": "stencil-95-k128-bf16", "op": "spmm", "matrix": "stencil27", "g": 95, "k": 128,
         "dtype": "f32", "storage": "bf16", "alpha": 1.0, "beta": 0.0},
        # Random sparse x dense in FP32 (features of a graph's nodes).
        {"name": "random-200k-k64-f32", "op": "spmm", "matrix": "uniform", "n": 200003, "ncols": 200003,
         "mean": 18, "k": 64, "dtype": "f32", "storage": "native", "alpha": 1.0, "beta": 0.0},
        # BSR x wide dense with BF16 values: the benchmark's block case.
        {"name": "bsr8-spmm-k128-bf16", "op": "bsr_spmm", "mb": 32768, "per_row": 8, "bs": 8,
         "rowmajor": True, "k": 128, "dtype": "f32", "storage": "bf16", "alpha": 1.0, "beta": 0.0},
        # Many independent uneven products in one launch (banded, random and
        # block-diagonal instances, as in the benchmark's batch).
        {"name": "batch-128-f32", "op": "batch", "count": 128, "sizes": 3, "alpha": 1.0, "beta": 0.0},
        # The drop-in call with vectors in (pinned) host memory.
        {"name": "host-laplace-1000-f64", "op": "spmv_host", "matrix": "laplace2d", "g": 1000,
         "dtype": "f64", "storage": "native", "optimize": True, "trans": False, "alpha": 1.0, "beta": 0.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scalars(rng):
    return rng.choice([(1.0, 0.0), (1.0, 0.0), (-0.75, 0.0), (1.5, 0.5)])


def _matrix(rng, n_max, nnz_max):
    """A matrix family with its sizes, at most n_max rows and nnz_max entries."""
    kind = rng.choice(["laplace2d", "stencil27", "zipf", "uniform", "banded"])
    if kind == "laplace2d":
        return {"matrix": kind, "g": _log(rng, 100, math.isqrt(n_max))}
    if kind == "stencil27":
        return {"matrix": kind, "g": _log(rng, 22, int(min(n_max, nnz_max // 27) ** (1 / 3) + 1e-9))}
    if kind == "zipf":
        return {"matrix": kind, "n": _log(rng, 10000, min(n_max, int(nnz_max / ZIPF_MEAN)))}
    if kind == "uniform":
        mean = _log(rng, 4, 32)
        n = _log(rng, 10000, min(n_max, nnz_max // mean))
        return {"matrix": kind, "n": n, "ncols": rng.choice([n, max(2000, int(n * rng.uniform(0.5, 1.5)))]),
                "mean": mean}
    hb = _log(rng, 2, 64)
    return {"matrix": kind, "n": _log(rng, 10000, min(n_max, nnz_max // (2 * hb + 1))), "hb": hb}


def draw(rng):
    op = rng.choice(["spmv", "spmv", "spmv", "bsr_spmv", "spmm", "spmm", "spmm", "bsr_spmm", "batch", "spmv_host"])
    alpha, beta = _scalars(rng)
    dtype = rng.choice(["f64", "f32"])
    storage = rng.choice(["native", "native", "fp32" if dtype == "f64" else "bf16", "bf16"])
    c = {"op": op, "alpha": alpha, "beta": beta}
    if op == "spmv":
        c.update(_matrix(rng, 2 ** 22, 48_000_000), dtype=dtype, storage=storage,
                 optimize=rng.random() < 0.5, trans=rng.random() < 0.25)
        if c["trans"]:
            c["optimize"] = True
    elif op == "spmv_host":
        c.update(_matrix(rng, 1_000_000, 16_000_000), dtype="f64", storage="native", optimize=True, trans=False)
    elif op == "bsr_spmv":
        bs = rng.choice([2, 4, 8])
        per = rng.randint(2, 16)
        mb = _log(rng, 2000, min(500_000, 40_000_000 // (per * bs * bs)))
        c.update(mb=mb, per_row=per, bs=bs, rowmajor=rng.random() < 0.5, dtype=dtype, storage=storage)
    elif op == "spmm":
        k = _log(rng, 6, 128)
        if rng.random() < 0.5:
            k = max(8, k // 8 * 8)
        c.update(_matrix(rng, min(2 ** 21, 64_000_000 // k), min(40_000_000, 500_000_000 // k)), k=k,
                 dtype=dtype, storage=storage)
    elif op == "bsr_spmm":
        bs = rng.choice([2, 4, 8])
        per = rng.randint(2, 12)
        k = _log(rng, 6, 128)
        if rng.random() < 0.5:
            k = max(8, k // 8 * 8)
        mb = _log(rng, 1000, min(32768 * 8 // bs, 400_000_000 // (per * bs * bs * k)))
        c.update(mb=mb, per_row=per, bs=bs, rowmajor=rng.random() < 0.5, k=k, dtype=dtype, storage=storage)
    else:
        c.update(count=_log(rng, 16, 128), sizes=rng.randint(10, 10 ** 6))
    return c


# ------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(shape, g, dtype=torch.float64):
    return torch.rand(shape, generator=g, device=DEV, dtype=dtype) * 2 - 1


def _from_lengths(lens, ncols, g):
    """Row pointers and sorted distinct uniform columns, about lens per row."""
    n = lens.numel()
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), lens)
    cols = torch.randint(ncols, (rows.numel(),), generator=g, device=DEV)
    key = torch.sort(rows.mul_(ncols).add_(cols)).values
    keep = torch.ones_like(key, dtype=torch.bool)
    keep[1:] = key[1:] != key[:-1]
    key = key[keep]
    counts = torch.bincount(key // ncols, minlength=n)
    rp = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rp[1:] = torch.cumsum(counts, 0)
    return rp, (key % ncols).to(torch.int32)


def _masked(cols, mask):
    rp = torch.zeros(cols.shape[0] + 1, dtype=torch.int32, device=DEV)
    rp[1:] = torch.cumsum(mask.sum(1), 0)
    return rp, cols[mask].to(torch.int32)


def _csr(case, g):
    """(rows, columns, row pointers, columns, FP64 values) on the GPU."""
    kind = case["matrix"]
    if kind == "laplace2d":
        s = case["g"]
        n = s * s
        i = torch.arange(n, device=DEV)
        r, c = i // s, i % s
        offs = ((-s, r > 0), (-1, c > 0), (0, r >= 0), (1, c < s - 1), (s, r < s - 1))
        mask = torch.stack([m for _, m in offs], 1)
        rp, col = _masked(torch.stack([i + o for o, _ in offs], 1), mask)
        v = torch.tensor([-1.0, -1.0, 4.0, -1.0, -1.0], dtype=torch.float64, device=DEV)
        return n, n, rp, col, v.expand(n, 5)[mask]
    if kind == "stencil27":
        s = case["g"]
        n = s ** 3
        i = torch.arange(n, device=DEV)
        z, y, x = i // (s * s), (i // s) % s, i % s
        cols, mask = [], []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    cols.append(i + (dz * s + dy) * s + dx)
                    mask.append((z + dz >= 0) & (z + dz < s) & (y + dy >= 0) & (y + dy < s)
                                & (x + dx >= 0) & (x + dx < s))
        mask = torch.stack(mask, 1)
        v = _uniform((n, 27), g)
        v[~mask] = 0
        v[:, 13] = 1 + v.abs().sum(1) - v[:, 13].abs()
        rp, col = _masked(torch.stack(cols, 1), mask)
        return n, n, rp, col, v[mask]
    if kind == "banded":
        n, hb = case["n"], case["hb"]
        cols = torch.arange(n, device=DEV)[:, None] + torch.arange(-hb, hb + 1, device=DEV)
        rp, col = _masked(cols, (cols >= 0) & (cols < n))
        return n, n, rp, col, _uniform(col.numel(), g)
    n = case["n"]
    if kind == "zipf":
        ncols = n
        k = torch.arange(1, ZIPF_MAX + 1, dtype=torch.float64, device=DEV)
        cdf = torch.cumsum((k + ZIPF_SHIFT) ** -2, 0)
        u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * cdf[-1]
        lens = (torch.searchsorted(cdf, u, right=True) + 1).clamp_(max=min(ZIPF_MAX, ncols))
        rp, col = _from_lengths(lens, ncols, g)
        return n, ncols, rp, col, torch.randn(col.numel(), generator=g, device=DEV, dtype=torch.float64)
    ncols, mean = case["ncols"], case["mean"]
    lens = torch.randint(max(1, mean // 2), mean + (mean + 1) // 2 + 1, (n,), generator=g, device=DEV)
    rp, col = _from_lengths(lens, ncols, g)
    return n, ncols, rp, col, _uniform(col.numel(), g)


def _bsr(case, g):
    """(rows, block row pointers, block columns, values [blocks, bs, bs] by row and column)."""
    mb, bs = case["mb"], case["bs"]
    rp, col = _from_lengths(torch.full((mb,), case["per_row"], device=DEV), mb, g)
    return mb * bs, rp, col, _uniform((col.numel(), bs, bs), g)


def _api(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _stored(v, case):
    """The values as the storage mode holds them, in FP64."""
    if case["dtype"] == "f32" or case["storage"] != "native":
        v = v.float()
    if case["storage"] == "bf16":
        v = v.to(torch.bfloat16)
    return v.double()


STORAGE = {"native": pls.STORAGE_NATIVE, "fp32": pls.STORAGE_FP32, "bf16": pls.STORAGE_BF16}


def _csr_handle(case, m, n, rp, col, v):
    if case["storage"] == "bf16":
        v = v.float()  # values that a double and a float round alike to BF16
    if case["dtype"] == "f64":
        v = v.double()
        A = pls.SpMat.csr_dev(m, n, rp.data_ptr(), col.data_ptr(), v.data_ptr())
    else:
        A = pls.SpMat.csr(m, n, rp.cpu().numpy(), col.cpu().numpy(), v.float().cpu().numpy())
    A.set_storage(STORAGE[case["storage"]])
    return A


def _bsr_handle(case, m, rp, col, v):
    np_v = (v if case["rowmajor"] else v.transpose(1, 2)).contiguous().to(_api(case)).cpu().numpy().reshape(-1)
    if case["storage"] == "bf16" and case["dtype"] == "f64":
        np_v = np_v.astype(np.float32).astype(np.float64)
    A = pls.SpMat.bsr(pls.ROW_MAJOR if case["rowmajor"] else pls.COL_MAJOR, m, m, case["bs"],
                      rp.cpu().numpy(), col.cpu().numpy(), np_v)
    A.set_storage(STORAGE[case["storage"]])
    return A


def _instances(case):
    """Sizes of a batch's instances, fixed by the case: kind, rows, k and what the kind needs."""
    r = random.Random(case["sizes"])
    out = []
    for i in range(case["count"]):
        n, k = _log(r, 1024, 65536), _log(r, 1, 64)
        kind = ("banded", "uniform", "bsr")[i % 3]
        d = {"kind": kind, "n": n, "k": k}
        if kind == "banded":
            d["hb"] = r.randint(2, 64)
        elif kind == "bsr":
            d["bs"] = r.choice([4, 8])
            d["n"] = n // d["bs"] * d["bs"]
            d["fill"] = r.uniform(0.3, 0.9)
        out.append(d)
    return out


def _batch_inputs(case, g):
    """Per instance (description, row pointers, columns, FP32 values), with all the dense
    operands in one buffer each, every operand on a 256-byte boundary."""
    inst, total = [], 0
    for d in _instances(case):
        n = d["n"]
        if d["kind"] == "bsr":
            nb = n // d["bs"]
            rp = torch.arange(nb + 1, dtype=torch.int32, device=DEV)
            col = rp[:-1].clone()
            v = _uniform((nb, d["bs"], d["bs"]), g, torch.float32)
            v = v * (torch.rand(v.shape, generator=g, device=DEV) < d["fill"])
        elif d["kind"] == "banded":
            _, _, rp, col, v = _csr({"matrix": "banded", "n": n, "hb": d["hb"]}, g)
        else:
            lens = torch.randint(4, 33, (n,), generator=g, device=DEV)
            rp, col = _from_lengths(lens, n, g)
            v = _uniform(col.numel(), g, torch.float32)
        inst.append((d, rp, col, v.float(), total))
        total += (n * d["k"] + 63) // 64 * 64
    B = _uniform(total, g, torch.float32)
    return inst, B


def prepare(case, seed):
    g = _gen(seed)
    op = case["op"]
    if op == "batch":
        inst, B = _batch_inputs(case, g)
        C = torch.zeros_like(B)
        mats = []
        for d, rp, col, v, _ in inst:
            rp, col, v = rp.cpu().numpy(), col.cpu().numpy(), v.cpu().numpy()
            if d["kind"] == "bsr":
                mats.append(pls.SpMat.bsr(pls.ROW_MAJOR, d["n"], d["n"], d["bs"], rp, col, v.reshape(-1)))
            else:
                mats.append(pls.SpMat.csr(d["n"], d["n"], rp, col, v))
        if case["beta"] != 0:
            C.copy_(_uniform(C.numel(), g, torch.float32))
        start = C.clone()
        ks = [d["k"] for d, *_ in inst]
        torch.cuda.synchronize()
        batch = pls.Batch(mats, ks, [B.data_ptr() + 4 * t for *_, t in inst], ks,
                          [C.data_ptr() + 4 * t for *_, t in inst], ks)
        batch.tune()  # the schedule a program picks once for its batch
        C.copy_(start)
        torch.cuda.synchronize()
        return {"case": case, "batch": batch, "mats": mats, "B": B, "C": C}
    k = case.get("k")
    if op in ("bsr_spmv", "bsr_spmm"):
        m, rp, col, v = _bsr(case, g)
        n = m
        A = _bsr_handle(case, m, rp, col, v)
    else:
        m, n, rp, col, v = _csr(case, g)
        A = _csr_handle(case, m, n, rp, col, v)
        del rp, col, v
    xl, yl = (m, n) if case.get("trans") else (n, m)
    x = _uniform(xl if k is None else (xl, k), g, _api(case))
    y = _uniform(yl if k is None else (yl, k), g, _api(case))
    if case.get("optimize"):
        if case["trans"]:
            A.hint(pls.HINT_SPMV_OPERATION, pls.OPERATION_TRANS)
        A.hint(pls.HINT_SPMV_INVOCATIONS, pls.INVOCATIONS_MANY)
        A.optimize()
    torch.cuda.synchronize()
    if k is not None:
        # The first product of a call signature picks its kernel; the handle keeps the choice.
        out = torch.empty_like(y)
        A.spmm_dev(x.data_ptr(), k, k, out.data_ptr(), k)
        torch.cuda.synchronize()
    if op == "spmv_host":
        x, y = x.cpu().pin_memory().numpy(), y.cpu().pin_memory().numpy()
    return {"case": case, "A": A, "x": x, "y": y, "k": k}


# ------------------------------------------------------------------ one pass

def run(s):
    case = s["case"]
    alpha, beta = case["alpha"], case["beta"]
    op = case["op"]
    if op == "batch":
        s["batch"].exec(alpha, beta)
        return s["C"]
    A, x, y, k = s["A"], s["x"], s["y"], s["k"]
    if op == "spmv_host":
        return A.spmv(x, y, alpha, beta)
    if k is not None:
        A.spmm_dev(x.data_ptr(), k, k, y.data_ptr(), k, alpha, beta)
    elif case.get("trans"):
        A.spmv_dev(x.data_ptr(), y.data_ptr(), alpha, beta, trans=pls.OPERATION_TRANS)
    else:
        A.spmv_dev(x.data_ptr(), y.data_ptr(), alpha, beta)
    return y


# ------------------------------------------------------------------ accounting

def _sizes(case):
    """(rows, columns, stored entries) of a case's matrix (about, where rows are drawn)."""
    kind = case["matrix"]
    if kind == "laplace2d":
        s = case["g"]
        return s * s, s * s, 5 * s * s - 4 * s
    if kind == "stencil27":
        s = case["g"]
        return s ** 3, s ** 3, (3 * s - 2) ** 3
    if kind == "banded":
        n, hb = case["n"], case["hb"]
        return n, n, n * (2 * hb + 1) - hb * (hb + 1)
    if kind == "zipf":
        return case["n"], case["n"], int(case["n"] * ZIPF_MEAN)
    return case["n"], case["ncols"], case["n"] * case["mean"]


def work(case):
    if case["op"] == "batch":
        nbytes = flops = 0
        for d in _instances(case):
            n, k = d["n"], d["k"]
            if d["kind"] == "bsr":
                nnz, index = n * d["bs"], n // d["bs"] * 8 + 4
            else:
                nnz = n * (2 * d["hb"] + 1) - d["hb"] * (d["hb"] + 1) if d["kind"] == "banded" else n * 18
                index = nnz * 4 + n * 4 + 4
            nbytes += nnz * 4 + index + n * k * 4 * (2 if case["beta"] == 0 else 3)
            flops += 2 * nnz * k
        return {"bytes": nbytes, "flops": flops}
    sx = 8 if case["dtype"] == "f64" else 4
    sv = {"native": sx, "fp32": 4, "bf16": 2}[case["storage"]]
    if case["op"].startswith("bsr"):
        bs = case["bs"]
        m = n = case["mb"] * bs
        nb = case["mb"] * case["per_row"]
        nnz, index = nb * bs * bs, nb * 4 + case["mb"] * 4 + 4
    else:
        m, n, nnz = _sizes(case)
        index = nnz * 4 + (m + 1) * 4
    if case.get("trans"):
        m, n = n, m
    k = case.get("k") or 1
    vectors = n * k + m * k * (1 if case["beta"] == 0 else 2)
    if case["op"] == "spmv_host":
        # the vectors cross the host link; the matrix is on the GPU
        return {"bytes": nnz * sv + index + vectors * sx, "flops": 2 * nnz}
    return {"bytes": nnz * sv + index + vectors * sx, "flops": 2 * nnz * k}


def tolerance(case):
    if case["op"] == "batch" or case["dtype"] == "f32" or case["storage"] != "native":
        # FP32 accumulation: sums in another order differ by a few 1e-7
        return {"rel": 1e-6, "max": 4e-5}
    return {"rel": 1e-14, "max": 1e-12}  # FP64 sums in another order, rows of up to 4096 terms


def _mul(m, n, rp, col, v, x, trans):
    if trans:
        rows = torch.repeat_interleave(torch.arange(m, device=DEV), rp.long().diff())
        return torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, col.long(), v * x[rows])
    A = torch.sparse_csr_tensor(rp, col, v, size=(m, n))
    return A @ x


def _expand(rp, col, v, bs):
    """The CSR arrays of a BSR matrix (every block entry kept)."""
    nb, mb = col.numel(), rp.numel() - 1
    brow = torch.repeat_interleave(torch.arange(mb, device=DEV), rp.long().diff())
    j = torch.arange(bs, device=DEV)
    pos = torch.arange(nb, device=DEV) - rp.long()[brow]
    width = rp.long().diff()
    # entry (block, i, jj) is number pos * bs + jj of row brow * bs + i
    srp = torch.zeros(mb * bs + 1, dtype=torch.int64, device=DEV)
    srp[1:] = torch.cumsum((width * bs).repeat_interleave(bs), 0)
    at = srp[(brow[:, None] * bs + j)][:, :, None] + (pos * bs)[:, None, None] + j
    cols = (col.long() * bs)[:, None, None] + j
    out_c = torch.empty(nb * bs * bs, dtype=torch.int32, device=DEV)
    out_v = torch.empty(nb * bs * bs, dtype=torch.float64, device=DEV)
    out_c[at.reshape(-1)] = cols.expand(nb, bs, bs).reshape(-1).to(torch.int32)
    out_v[at.reshape(-1)] = v.reshape(-1)
    return srp.to(torch.int32), out_c, out_v


def exact(case, seed):
    g = _gen(seed)
    alpha, beta = case["alpha"], case["beta"]
    if case["op"] == "batch":
        inst, B = _batch_inputs(case, g)
        C = torch.zeros(B.numel(), dtype=torch.float64, device=DEV)
        if beta != 0:
            C += _uniform(C.numel(), g, torch.float32).double()
        for d, rp, col, v, t in inst:
            n, k = d["n"], d["k"]
            if d["kind"] == "bsr":
                rp, col, v = _expand(rp, col, v.double(), d["bs"])
            part = slice(t, t + n * k)
            ab = _mul(n, n, rp, col, v.double(), B[part].double().view(n, k), False)
            C[part] = alpha * ab.reshape(-1) + beta * C[part]
        return C
    k = case.get("k")
    if case["op"].startswith("bsr"):
        m, rp, col, v = _bsr(case, g)
        n = m
        rp, col, v = _expand(rp, col, v, case["bs"])
    else:
        m, n, rp, col, v = _csr(case, g)
    trans = bool(case.get("trans"))
    xl, yl = (m, n) if trans else (n, m)
    x = _uniform(xl if k is None else (xl, k), g, _api(case)).double()
    y = _uniform(yl if k is None else (yl, k), g, _api(case)).double()
    out = alpha * _mul(m, n, rp, col, _stored(v, case), x, trans)
    if beta != 0:
        out += beta * y
    return out.cpu().numpy() if case["op"] == "spmv_host" else out
