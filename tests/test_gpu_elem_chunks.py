"""COO plans, and BCOO plans of 2x2, 4x4 and 8x8 blocks, which run in staged
chunks whose first and last rows may be shared with the neighbouring chunks:
sizes around a chunk, rows over one to many chunks (more than a warp's worth of
parts to add), rows of one nonzero, gaps of empty rows, cuts off the copies'
alignment, warps per CTA, atomics, tiles.  Each plan runs twice (the arrival
counters start again).  Integers bit for bit, FP within gamma_n sum|a x|."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi
from helpers import fp_bound_ok, hi_ref, random_x

pytestmark = pytest.mark.gpu


def check(y, nrows, r, c, v, x, dtype):
    if np.dtype(capi.DTYPES[dtype].np).kind == "f":
        ok, err, bound = fp_bound_ok(y, *hi_ref(r, c, v, x, nrows), dtype)
        assert ok, float((err / bound).max())
    else:
        want = np.zeros(nrows, np.uint64)
        np.add.at(want, r, v.astype(np.int64).astype(np.uint64) * x[c].astype(np.int64).astype(np.uint64))
        assert np.array_equal(y, want.astype(capi.DTYPES[dtype].np))


def twice(plan, *want):
    for _ in range(2):
        check(plan.run_host(want[4]), *want)


def lengths(rng, kind):
    if isinstance(kind, int):  # nonzeros in all, rows of 0..3
        lens = rng.integers(0, 4, kind + 3)
        lens[np.cumsum(lens) > kind] = 0
        lens[-1] = kind - lens.sum()
        return lens
    if kind == "long":
        return np.array([5, 0, 2043, 1, 4097, 0, 0, 90_001, 1, 1, 2047, 6000, 0, 3])
    return np.concatenate([np.ones(3000, int), np.zeros(400, int), rng.integers(0, 60, 500), np.zeros(70, int)])


@pytest.mark.parametrize("dtype", list(capi.DTYPES))
@pytest.mark.parametrize("kind", [0, 1, 2047, 2048, 2049, 6145, "long", "mixed"])
def test_coo(dtype, kind):
    rng = np.random.default_rng(11)
    lens = lengths(rng, kind)
    nrows, ncols = lens.size, 3001
    r = np.repeat(np.arange(nrows, dtype=np.uint32), lens)
    c = rng.integers(0, ncols, r.size).astype(np.uint32)
    c = c[np.lexsort((c, r))]
    v, x = random_x(rng, r.size, dtype), random_x(rng, ncols, dtype)
    A = sp.cooe(dtype, nrows, ncols, r, c, v)
    for o in (dict(), dict(nr_workers=1), dict(nr_workers=16), dict(nr_parts=3, part_balance=capi.BAL_NNZ_ELEM),
              dict(nr_parts=5, part_balance=capi.BAL_ROW), dict(sync=capi.SYNC_ATOMIC)):
        twice(sp.Plan(A, sp.default_opts(**o)), nrows, r, c, v, x, dtype)
    if dtype in ("f32", "i8"):
        for conv in ("cooe2dcoo", "cooe2bdcoo"):
            for st in (0, 1):
                D = sp.convert(conv, A, 3, 2)
                twice(sp.Plan(D, sp.default_opts(stage_x=st)), nrows, r, c, v, x, dtype)


@pytest.mark.parametrize("dtype", list(capi.DTYPES))
@pytest.mark.parametrize("b", [2, 4, 8])
def test_bcoo(dtype, b):
    rng = np.random.default_rng(b)
    chunk = min(1024, 32768 // (b * b * np.dtype(capi.DTYPES[dtype].np).itemsize))
    nbc = 5 * chunk + 9
    counts = np.concatenate([[0, 0, 3, 4 * chunk + 7, 0, chunk - 5, 1, chunk, 0], rng.integers(0, 30, 60),
                             np.ones(chunk + 40, int), [0, 5 * chunk, 2, 0, 0]])
    nbr = counts.size
    nrows, ncols = nbr * b - 1, nbc * b - 1
    browptr = np.zeros(nbr + 1, np.uint32)
    np.cumsum(counts, out=browptr[1:])
    bcol = np.concatenate([np.sort(rng.choice(nbc, n, replace=False)) for n in counts]).astype(np.uint32)
    bval = random_x(rng, bcol.size * b * b, dtype).reshape(-1, b, b)
    bval[bcol == nbc - 1, :, b - 1] = 0
    B = dict(nrows=nrows, ncols=ncols, rb=b, cb=b, nbr=nbr, browptr=browptr, bcolind=bcol, bval=bval)
    r, c, v = sp.synth.bcsr_triplets(B)
    x = random_x(rng, ncols, dtype)
    A = sp.convert("bcsr2bcoo", capi.bcsr(dtype, nrows, ncols, b, b, browptr, bcol, bval, int((bval != 0).sum())))
    for o in (dict(), dict(lanes=1, nr_workers=1), dict(nr_workers=16), dict(nr_parts=7),
              dict(nr_parts=9, part_balance=capi.BAL_BLOCK), dict(sync=capi.SYNC_ATOMIC)):
        twice(sp.Plan(A, sp.default_opts(**o)), nrows, r, c, v, x, dtype)
    o = np.lexsort((c, r))
    o = o[v[o] != 0]
    D = sp.convert("dcsr2dbcoo", sp.convert("cooe2dcsr", sp.cooe(dtype, nrows, ncols, r[o], c[o], v[o]), 2, 3), b, b)
    for st in (0, 1):
        twice(sp.Plan(D, sp.default_opts(stage_x=st)), nrows, r, c, v, x, dtype)
