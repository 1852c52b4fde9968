"""The work that users of sparsep_b200 have it do, as measurable cases.

Every case goes through the public entry points: a plan over a host or device
matrix and its execution on device or host buffers, the batched multi-RHS
launch, the device format converters, conjugate gradient on a plan.  Sizes are
those of the benchmark workloads (the 4096-row uniform matrix, the 1M-row
power-law matrix with mean row length 16, the 2M-row block-banded matrix, the
mixed batch of small and large matrices, the 1M-unknown Laplacian) or ragged
neighbours of them; draw() spreads over the same ranges.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import sparsep_b200 as sp
from sparsep_b200 import capi, selector

TORCH = {"i8": torch.int8, "i16": torch.int16, "i32": torch.int32, "i64": torch.int64, "f32": torch.float32,
         "f64": torch.float64}
SIZE = {"i8": 1, "i16": 2, "i32": 4, "i64": 8, "f32": 4, "f64": 8}
HALF_BW = 32  # block half-bandwidth of the block-banded pattern
TILED = ("dcsr", "rbdcsr", "bdcsr", "dcoo", "rbdcoo", "bdcoo")


def spmv(name, fmt, dtype, pattern, rows, nnz, **kw):
    return dict(name=name, op="spmv", format=fmt, dtype=dtype, pattern=pattern, rows=rows, cols=kw.pop("cols", rows),
                nnz=nnz, **{"parts": 0, "sync": "lf", "via": "device", "grid": 0, **kw})


def blocks(name, fmt, dtype, rows, block, per_row, parts=0):
    return dict(name=name, op="block", format=fmt, dtype=dtype, rows=rows, block=block, per_row=per_row, parts=parts)


def listed():
    return [
        # one call on a small matrix: launch and latency
        spmv("csr i32 4k", "csr", "i32", "uniform", 4096, 8 * 4096),
        # the library's headline: a power-law graph in CSR, single precision, vectors on the device
        spmv("csr f32 1M", "csr", "f32", "zipf", 1 << 20, 16 << 20),
        # the same in double precision, as scientific codes run it, at a ragged size
        spmv("csr f64 1M", "csr", "f64", "zipf", 999_983, 15_999_728),
        # one call on the caller's host vectors, copies included
        spmv("host f32 786k", "csr", "f32", "zipf", 786_433, 12_582_912, via="host"),
        # coordinate format, as an edge list comes
        spmv("coo f32 1M", "coo", "f32", "zipf", 1 << 20, 16 << 20),
        # the reference's 2D partitioning: equal tiles, partial results merged
        spmv("2d dcoo f32 524k", "dcoo", "f32", "zipf", 524_309, 8_388_944, grid=16),
        # finite-element style matrices stored in dense blocks
        blocks("bcsr f32 4x4 2M", "bcsr", "f32", 1 << 21, 4, 20),
        blocks("bcsr i8 8x8 2M", "bcsr", "i8", 1 << 21, 8, 20, parts=2048),
        blocks("bcoo i16 4x4 1M", "bcoo", "i16", 1_000_006, 4, 20),
        # many matrices of mixed sizes, each with its own right-hand sides, in one launch
        dict(name="batch f32 48", op="batch", dtype="f32", mats=48, rows_lo=1_000, rows_hi=256_000, k_max=32),
        # ingest on the device: an unsorted edge list to CSR and on to blocks
        dict(name="convert f32 10M", op="convert", dtype="f32", rows=1 << 19, block=4, per_row=8),
        # an iterative solver around the product: the 5-point Laplacian
        dict(name="cg f64 1M", op="cg", dtype="f64", side=1024, iters=25),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["csr", "csr", "coo", "2d", "bcsr", "bcoo", "batch", "convert", "cg"])
    dtype = rng.choice(["i8", "i16", "i32", "i64", "f32", "f32", "f64"])
    if op in ("csr", "coo", "2d"):
        rows = log_int(rng, 4_096, 1 << 20)
        nnz = min(16 << 20, int(rows * math.exp(rng.uniform(math.log(4), math.log(64)))))
        pattern = rng.choice(["uniform", "zipf", "banded"])
        cols = rows if pattern == "banded" else log_int(rng, max(4_096, rows // 2), 2 * rows)
        kw = dict(cols=cols)
        if op == "2d":
            op, kw["grid"] = rng.choice(TILED), rng.choice([4, 8, 16, 32])
        else:
            kw["parts"] = rng.choice([0, 0, 0, 2048])
            kw["via"] = rng.choice(["device", "device", "host"])
        if op != "csr":
            kw["sync"] = rng.choice(["lf", "lf", "atomic"])
        c = spmv("", op, dtype, pattern, rows, nnz, **kw)
    elif op in ("bcsr", "bcoo"):
        b = rng.choice([2, 4, 8])
        per_row = rng.randint(4, 24)
        most = min((1 << 27) // (per_row * b * SIZE[dtype]), 1 << 21)  # at most half a gigabyte of blocks
        c = blocks("", op, dtype, log_int(rng, 16_384, most), b, per_row, rng.choice([0, 2048]))
    elif op == "batch":
        c = dict(op="batch", dtype=rng.choice(["f32", "i32"]), mats=rng.randint(8, 48), rows_lo=1_000,
                 rows_hi=log_int(rng, 16_000, 256_000), k_max=rng.randint(1, 32))
    elif op == "convert":
        b = rng.choice([2, 4])
        c = dict(op="convert", dtype=dtype, rows=b * log_int(rng, 4_096, (1 << 19) // b), block=b,
                 per_row=rng.randint(3, 8))  # whole blocks: every list of the same size fills as many
    else:
        c = dict(op="cg", dtype=rng.choice(["f32", "f64"]), side=rng.randint(100, 1024), iters=rng.randint(5, 25))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def values(g, n, dtype):
    """Uniform in [-1, 1], or integers in [-8, 8]."""
    t = TORCH[dtype]
    if t.is_floating_point:
        return torch.rand(n, device="cuda", generator=g, dtype=t) * 2 - 1
    return torch.randint(-8, 9, n if isinstance(n, tuple) else (n,), device="cuda", generator=g).to(t)


@functools.lru_cache(maxsize=256)
def row_lengths(pattern, rows, cols, nnz):
    """The row lengths of a pattern, nnz in all, in an order that the seed then
    permutes.  uniform: 8 per row where nnz is 8 per row, else spread over
    [m/2, 3m/2]; zipf: power law with exponent 2, capped at 50,000; banded: as uniform."""
    mean = nnz / rows
    most = min(cols, 50_000)
    if pattern == "zipf":
        z = np.minimum(np.random.default_rng(rows).zipf(2.0, rows), 50_000).astype(np.float64)
        lens = np.maximum(1, np.floor(z * (nnz / z.sum()))).astype(np.int64)
    elif mean == 8:
        lens = np.full(rows, 8, dtype=np.int64)
    else:
        lens = np.floor(np.linspace(mean / 2, 3 * mean / 2, rows)).astype(np.int64)
    lens = np.clip(lens, 1, most)
    while (d := nnz - int(lens.sum())) != 0:  # hand the rounding's rest to rows that have room
        at = np.nonzero(lens < most if d > 0 else lens > 1)[0]
        at = at[:: max(1, at.size // abs(d))][: abs(d)]
        lens[at] += 1 if d > 0 else -1
    return lens


def band_width(rows, nnz):
    return int(min(rows, 8 * math.ceil(nnz / rows) + 1))


def pattern_csr(g, pattern, rows, cols, nnz):
    """rowptr, row of each nonzero and sorted distinct columns: one draw inside each
    of a row's equal strata of [0, cols), or of its band."""
    lens = torch.from_numpy(row_lengths(pattern, rows, cols, nnz)).cuda()
    lens = lens[torch.randperm(rows, device="cuda", generator=g)]
    rowptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=rowptr[1:])
    row = torch.repeat_interleave(torch.arange(rows, device="cuda"), lens, output_size=nnz)
    i = torch.arange(nnz, device="cuda") - rowptr[row]
    ln = lens[row]
    lo, width = 0, cols
    if pattern == "banded":
        width = band_width(rows, nnz)
        lo = torch.clamp(row - width // 2, 0, rows - width)
    a = i * width // ln
    span = (i + 1) * width // ln - a
    u = torch.rand(nnz, device="cuda", generator=g, dtype=torch.float64)
    col = lo + a + torch.minimum((u * span).long(), span - 1)
    return rowptr, row, col


def spmv_inputs(c, seed):
    g = generator(seed)
    rowptr, row, col = pattern_csr(g, c["pattern"], c["rows"], c["cols"], c["nnz"])
    return rowptr, row, col, values(g, c["nnz"], c["dtype"]), values(g, c["cols"], c["dtype"])


def block_geometry(c):
    nbr = -(-c["rows"] // c["block"])
    return nbr, min(c["per_row"], nbr, HALF_BW + 1)


def block_pattern(g, nbr, per):
    """Sorted block columns of each block row: `per` of its band, (nbr, per)."""
    out = torch.empty(nbr, per, dtype=torch.int64, device="cuda")
    for a in range(0, nbr, 1 << 17):
        i = torch.arange(a, min(nbr, a + (1 << 17)), device="cuda")
        j = i[:, None] + torch.arange(-HALF_BW, HALF_BW + 1, device="cuda")[None, :]
        u = torch.rand(j.shape, device="cuda", generator=g).masked_fill_((j < 0) | (j >= nbr), -1.0)
        out[a : a + i.numel()] = torch.gather(j, 1, u.topk(per, 1).indices).sort(1).values
    return out


def block_inputs(c, seed):
    """Block columns (nbr, per), dense blocks 60% full, zero past the last row and column, and x."""
    g = generator(seed)
    b, rows = c["block"], c["rows"]
    nbr, per = block_geometry(c)
    bcol = block_pattern(g, nbr, per)
    bval = torch.empty(nbr * per, b, b, dtype=TORCH[c["dtype"]], device="cuda")
    step = max(1, (1 << 25) // (b * b))
    for a in range(0, nbr * per, step):
        part = bval[a : a + step]
        v = values(g, tuple(part.shape), c["dtype"])
        part.copy_(v * (torch.rand(part.shape, device="cuda", generator=g) < 0.6))
    if rows % b:
        bval.view(nbr, per, b, b)[-1, :, rows % b :, :] = 0
        bval[bcol.reshape(-1) == nbr - 1, :, rows % b :] = 0
    return bcol, bval, values(g, rows, c["dtype"])


def batch_shapes(c):
    """(pattern, rows, nnz, k) of each matrix: rows spread over their logarithm, patterns and k in turn."""
    m, out = c["mats"], []
    for i in range(m):
        j = (i * 29) % m  # sizes in mixed order
        n = int(c["rows_lo"] * (c["rows_hi"] / c["rows_lo"]) ** (j / max(1, m - 1)))
        pattern = ("uniform", "zipf", "banded")[i % 3]
        out.append((pattern, n, n * (16 if pattern == "zipf" else 34), 1 + (i * 11) % c["k_max"]))
    return out


def batch_inputs(c, seed):
    g = generator(seed)
    for pattern, n, nnz, k in batch_shapes(c):
        rowptr, row, col = pattern_csr(g, pattern, n, n, nnz)
        yield rowptr, row, col, values(g, nnz, c["dtype"]), values(g, (n, k), c["dtype"])


def convert_inputs(c, seed):
    """An unsorted coordinate list whose blocks hold 10 of 16 (or 2 of 4) entries."""
    g = generator(seed)
    b = c["block"]
    nbr, per = block_geometry(c)
    bcol = block_pattern(g, nbr, per).reshape(-1)
    brow = torch.arange(nbr, device="cuda").repeat_interleave(per)
    fill = torch.rand(nbr * per, b * b, device="cuda", generator=g).topk(10 if b == 4 else 2, 1).indices
    row = (brow[:, None] * b + fill // b).reshape(-1)
    col = (bcol[:, None] * b + fill % b).reshape(-1)
    order = torch.randperm(row.numel(), device="cuda", generator=g)
    return row[order].int(), col[order].int(), values(g, row.numel(), c["dtype"])


def laplacian(side, dtype):
    """CSR of the shifted 5-point Laplacian on a side x side grid."""
    n = side * side
    i = torch.arange(n, device="cuda")
    y, x = i // side, i % side
    at = torch.stack([i - side, i - 1, i, i + 1, i + side], 1)
    ok = torch.stack([y > 0, x > 0, torch.ones_like(i, dtype=torch.bool), x < side - 1, y < side - 1], 1)
    val = torch.tensor([-1.0, -1.0, 4.05, -1.0, -1.0], dtype=TORCH[dtype], device="cuda").expand(n, 5)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(ok.sum(1), 0, out=rowptr[1:])
    return rowptr, at[ok], val[ok].contiguous()


# ---------------------------------------------------------------------------
# state and pass
# ---------------------------------------------------------------------------
def numpy32(t):
    return t.int().cpu().numpy().view(np.uint32)


def host_csr(c, dtype, rows, cols, rowptr, col, val):
    return sp.csr(dtype, rows, cols, numpy32(rowptr), numpy32(col), val.cpu().numpy())


class OnDevice:
    """A device buffer of `owner` as an array; a tensor made of it keeps the owner alive."""

    def __init__(self, owner, ptr, shape, dtype):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "version": 3,
                                         "typestr": {"f32": "<f4", "i32": "<i4"}[dtype]}


def prepare_spmv(c, seed):
    rowptr, row, col, val, x = spmv_inputs(c, seed)
    rows, cols, fmt, dtype = c["rows"], c["cols"], c["format"], c["dtype"]
    if fmt == "csr":
        A = host_csr(c, dtype, rows, cols, rowptr, col, val)
    else:
        A = sp.cooe(dtype, rows, cols, numpy32(row), numpy32(col), val.cpu().numpy())
        if fmt in TILED:
            A = sp.convert("cooe2" + fmt, A, c["grid"], c["grid"])
    o = sp.default_opts(nr_parts=c["parts"], part_balance=capi.BAL_NNZ,
                        sync=capi.SYNC_ATOMIC if c["sync"] == "atomic" else capi.SYNC_LF)
    s = {"plan": sp.Plan(A, o)}
    s["plan"].A = None  # the plan holds its own copy on the device
    if c["via"] == "host":
        s["x"], s["y"] = x.cpu().pin_memory(), torch.empty(rows, dtype=TORCH[dtype]).pin_memory()
    else:
        s["x"], s["y"] = x, torch.empty(rows, dtype=TORCH[dtype], device="cuda")
    return s


def prepare_block(c, seed):
    bcol, bval, x = block_inputs(c, seed)
    rows, b, dtype = c["rows"], c["block"], c["dtype"]
    nbr, per = bcol.shape
    browptr = torch.arange(nbr + 1, device="cuda", dtype=torch.int32) * per
    npb = (bval != 0).sum((1, 2), dtype=torch.int32)
    nnz = int(npb.sum())
    o = sp.default_opts(nr_parts=c["parts"], part_balance=capi.BAL_BLOCK, row_block_size=b, col_block_size=b)
    if c["format"] == "bcsr":
        bcol32 = bcol.reshape(-1).int()
        plan = sp.Plan.from_device_bcsr(dtype, rows, rows, b, b, nbr * per, nnz, browptr.data_ptr(), bcol32.data_ptr(),
                                        bval.data_ptr(), npb.data_ptr(), o)
    else:
        A = capi.bcsr(dtype, rows, rows, b, b, numpy32(browptr), numpy32(bcol.reshape(-1)), bval.cpu().numpy(), nnz,
                      numpy32(npb))
        plan = sp.Plan(sp.convert("bcsr2bcoo", A), o)
        plan.A = None
    return {"plan": plan, "x": x, "y": torch.empty(rows, dtype=TORCH[dtype], device="cuda")}


def prepare_batch(c, seed):
    mats, xs = [], []
    for rowptr, _, col, val, x in batch_inputs(c, seed):
        mats.append(host_csr(c, c["dtype"], x.shape[0], x.shape[0], rowptr, col, val))
        xs.append(x.cpu().numpy())
    batch = capi.Batch(c["dtype"], mats, [x.shape[1] for x in xs])
    batch.select(selector.selector(selector.load()))
    for m, x in enumerate(xs):
        batch.set_x(m, x)
    y = []
    for m, x in enumerate(xs):
        rows = OnDevice(batch, batch.device_xy(m)[1], (x.shape[0], batch.pitch(m)), c["dtype"])
        y.append(torch.as_tensor(rows, device="cuda")[:, : x.shape[1]])
    return {"batch": batch, "y": y, "stream": torch.cuda.Stream()}


def prepare_convert(c, seed):
    row, col, val = convert_inputs(c, seed)
    f = getattr(sp.lib(), "sparsep_coo2csr_device_" + c["dtype"])
    f.argtypes = [C.c_void_p] * 3 + [C.c_uint32] * 2 + [C.c_void_p] * 4
    return {"coo": (row, col, val), "coo2csr": f}


def prepare_cg(c, seed):
    n = c["side"] ** 2
    rowptr, col, val = laplacian(c["side"], c["dtype"])
    rowptr, col = rowptr.int(), col.int()
    plan = sp.Plan.from_device_csr(c["dtype"], n, n, col.numel(), rowptr.data_ptr(), col.data_ptr(), val.data_ptr())
    return {"cg": capi.CG(plan), "b": values(generator(seed), n, c["dtype"]),
            "x": torch.empty(n, dtype=TORCH[c["dtype"]], device="cuda")}


def prepare(case, seed):
    s = {"spmv": prepare_spmv, "block": prepare_block, "batch": prepare_batch, "convert": prepare_convert,
         "cg": prepare_cg}[case["op"]](case, seed)
    s["case"] = case
    return s


def run(s):
    c = s["case"]
    stream = torch.cuda.current_stream().cuda_stream
    if c["op"] in ("spmv", "block"):
        if c.get("via") == "host":
            capi.check(sp.lib().sparsep_execute_host(s["plan"].h, s["x"].data_ptr(), s["y"].data_ptr()))
        else:
            s["plan"].run_device(s["x"].data_ptr(), s["y"].data_ptr(), stream)
        return s["y"]
    if c["op"] == "batch":
        s["batch"].execute(s["stream"].cuda_stream)
        return s["y"]
    if c["op"] == "cg":
        s["x"].zero_()
        s["cg"].solve(s["b"].data_ptr(), s["x"].data_ptr(), max_iters=c["iters"], rel_tol=0.0, check_every=c["iters"],
                      stream=stream)
        return s["x"]
    row, col, val = s["coo"]
    n, b, nnz = c["rows"], c["block"], val.numel()
    i32 = dict(dtype=torch.int32, device="cuda")
    rowptr, colind, v = torch.empty(n + 1, **i32), torch.empty(nnz, **i32), torch.empty_like(val)
    capi.check(s["coo2csr"](row.data_ptr(), col.data_ptr(), val.data_ptr(), nnz, n, rowptr.data_ptr(),
                            colind.data_ptr(), v.data_ptr(), stream), "coo2csr_device")
    layout = capi.BcsrLayout(rowptr.data_ptr(), colind.data_ptr(), n, n, nnz, b, b, stream)
    browptr, bcolind = torch.empty(layout.nbr + 1, **i32), torch.empty(layout.nblocks, **i32)
    bval, npb = torch.empty(layout.nblocks, b, b, dtype=val.dtype, device="cuda"), torch.empty(layout.nblocks, **i32)
    layout.fill(c["dtype"], v.data_ptr(), browptr.data_ptr(), bcolind.data_ptr(), bval.data_ptr(), npb.data_ptr(),
                stream)
    layout.free()
    return {"rowptr": rowptr, "colind": colind, "values": v, "browptr": browptr, "bcolind": bcolind, "bval": bval,
            "nnz_per_block": npb}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its results in 64 bits
# ---------------------------------------------------------------------------
def work(c):
    if c["op"] == "batch":
        s, b, f = SIZE[c["dtype"]], 0, 0
        for _, n, nnz, k in batch_shapes(c):
            b += nnz * (4 + s) + (n + 1) * 4 + 2 * n * k * s
            f += 2 * nnz * k
        return {"bytes": b, "flops": f}
    if c["op"] == "cg":
        n, s = c["side"] ** 2, SIZE[c["dtype"]]
        nnz = 5 * n - 4 * c["side"]
        # per iteration the matrix once, p and q of the product, and x, r, p read and written with q read again
        return {"bytes": (c["iters"] + 1) * (nnz * (4 + s) + 4 * n + 2 * n * s) + c["iters"] * 7 * n * s,
                "flops": (c["iters"] + 1) * 2 * nnz + c["iters"] * 10 * n}
    s = SIZE[c["dtype"]]
    if c["op"] == "spmv":
        idx = c["nnz"] * 4 + (c["rows"] + 1) * 4 if c["format"].endswith("csr") else c["nnz"] * 8
        return {"bytes": idx + (c["nnz"] + c["rows"] + c["cols"]) * s, "flops": 2 * c["nnz"]}
    nbr, per = block_geometry(c)
    nb, b = nbr * per, c["block"]
    if c["op"] == "block":
        idx = nb * 4 + (nbr + 1) * 4 if c["format"] == "bcsr" else nb * 8
        return {"bytes": idx + (nb * b * b + 2 * c["rows"]) * s, "flops": 2 * nb * b * b}
    nnz = nb * (10 if b == 4 else 2)
    # the list read, the CSR written and read again, the blocks written
    return {"bytes": nnz * (8 + s) + 2 * (nnz * (4 + s) + 4 * c["rows"]) + nb * (b * b * s + 8) + 4 * nbr,
            "flops": 0}


def wide(t):
    return t.double() if t.is_floating_point() else t.long()


def in_type(y, dtype):
    """64-bit sums: as they are, or wrapped to the integer type."""
    return y if TORCH[dtype].is_floating_point else y.to(TORCH[dtype])


def product(rows, row, col, val, x):
    y = torch.zeros((rows,) + tuple(x.shape[1:]), dtype=wide(x[:1]).dtype, device="cuda")
    for a in range(0, row.numel(), 1 << 22):
        e = a + (1 << 22)
        v = wide(val[a:e])
        y.index_add_(0, row[a:e], (v[:, None] if x.dim() > 1 else v) * wide(x[col[a:e]]))
    return y


def exact(c, seed):
    if c["op"] == "spmv":
        _, row, col, val, x = spmv_inputs(c, seed)
        y = in_type(product(c["rows"], row, col, val, x), c["dtype"])
        return y.cpu() if c["via"] == "host" else y
    if c["op"] == "batch":
        return [in_type(product(x.shape[0], row, col, val, x), c["dtype"])
                for _, row, col, val, x in batch_inputs(c, seed)]
    if c["op"] == "block":
        bcol, bval, x = block_inputs(c, seed)
        nbr, per = bcol.shape
        b, rows = c["block"], c["rows"]
        xp = torch.zeros(nbr * b, dtype=wide(x[:1]).dtype, device="cuda")
        xp[:rows] = x
        y = torch.zeros(nbr, b, dtype=xp.dtype, device="cuda")
        for j in range(per):
            y += (wide(bval.view(nbr, per, b, b)[:, j]) * xp.view(nbr, b)[bcol[:, j]][:, None, :]).sum(2)
        return in_type(y.reshape(-1)[:rows], c["dtype"])
    if c["op"] == "cg":
        side = c["side"]
        b = wide(values(generator(seed), side * side, c["dtype"])).view(side, side)
        diagonal = 4.05 if c["dtype"] == "f64" else float(np.float32(4.05))

        def mul(p):
            q = diagonal * p
            q[1:] -= p[:-1]
            q[:-1] -= p[1:]
            q[:, 1:] -= p[:, :-1]
            q[:, :-1] -= p[:, 1:]
            return q

        x, r, p = torch.zeros_like(b), b.clone(), b.clone()
        rr = (r * r).sum()
        for _ in range(c["iters"]):
            q = mul(p)
            alpha = rr / (p * q).sum()
            x, r = x + alpha * p, r - alpha * q
            rr, last = (r * r).sum(), rr
            p = r + rr / last * p
        return x.reshape(-1)
    row, col, val = convert_inputs(c, seed)
    n, b = c["rows"], c["block"]
    nbr, per = block_geometry(c)
    order = torch.sort(row, stable=True).indices
    row, col, val = row[order].long(), col[order].long(), wide(val[order])
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(row, minlength=n), 0, out=rowptr[1:])
    key, inverse = torch.unique(row // b * nbr + col // b, return_inverse=True)
    bval = torch.zeros(key.numel(), b, b, dtype=val.dtype, device="cuda")
    bval[inverse, row % b, col % b] = val
    browptr = torch.arange(nbr + 1, device="cuda") * per
    i32 = torch.int32
    return {"rowptr": rowptr.to(i32), "colind": col.to(i32), "values": in_type(val, c["dtype"]),
            "browptr": browptr.to(i32), "bcolind": (key % nbr).to(i32), "bval": in_type(bval, c["dtype"]),
            "nnz_per_block": (bval != 0).sum((1, 2), dtype=i32)}
