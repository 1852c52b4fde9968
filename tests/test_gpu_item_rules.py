"""The rules by which plans choose their items, at both sides of their lines: lanes of
BCSR chunks with few block rows, the row kernel's two forms by row length and warps,
COO items by warps and atomics.  Integers bit for bit, FP within gamma_n sum|a x|."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi
from helpers import random_x
from test_gpu_elem_chunks import check
from test_gpu_elem_gaps import run

pytestmark = pytest.mark.gpu


def matrix(dtype, lens, ncols=5003, seed=1):
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(lens.size, dtype=np.uint32), lens)
    c = rng.integers(0, ncols, r.size).astype(np.uint32)
    c = c[np.lexsort((c, r))]
    return lens.size, r, c, random_x(rng, r.size, dtype), random_x(rng, ncols, dtype), dtype


def csr(want):
    nrows, r, c, v, x, dtype = want
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=nrows))]).astype(np.uint32)
    return sp.csr(dtype, nrows, x.size, rowptr, c, v)


def items(A, want, **o):
    """Items of the plan, whose results are checked twice."""
    plan = sp.Plan(A, sp.default_opts(**o))
    for _ in range(2):
        check(run(plan, want[4], want[0]), *want)
    n = int(plan.info.items)
    plan.free()
    return n


@pytest.mark.parametrize("dtype", ["i8", "i16", "f32", "f64"])
@pytest.mark.parametrize("b", [4, 8])
@pytest.mark.parametrize("per", [1, 3, 20])
def test_few_block_rows_take_more_lanes(dtype, b, per):
    rng = np.random.default_rng(per)
    for nbr in (1, 60, 700):
        ncb = 40
        bcol = np.concatenate([np.sort(rng.choice(ncb, per, replace=False)) for _ in range(nbr)]).astype(np.uint32)
        bval, x = random_x(rng, nbr * per * b * b, dtype), random_x(rng, ncb * b, dtype)
        A = capi.bcsr(dtype, nbr * b, ncb * b, b, b, np.arange(nbr + 1) * per, bcol, bval, bval.size,
                      np.full(nbr * per, b * b, np.uint32))
        row = np.repeat(np.arange(nbr), per)[:, None, None] * b + np.arange(b)[None, :, None] + np.zeros((1, 1, b), int)
        col = bcol.astype(int)[:, None, None] * b + np.arange(b)[None, None, :] + np.zeros((1, b, 1), int)
        plan = sp.Plan(A)
        for _ in range(2):
            check(run(plan, x, nbr * b), nbr * b, row.reshape(-1).astype(np.uint32), col.reshape(-1).astype(np.uint32),
                  bval, x, dtype)
        if per == 20 and b * b * bval.itemsize <= 128:  # 4 block rows per chunk: room for 8 lane groups each
            assert plan.info.lanes == 8 and plan.info.items >= nbr / 4
        plan.free()


@pytest.mark.parametrize("dtype", ["i16", "f32"])
@pytest.mark.parametrize("b", [2, 4, 8])
def test_parts_smaller_than_a_chunk_share_it(dtype, b):
    rng = np.random.default_rng(b)
    nbr, ncb = 3000, 40
    per = rng.integers(0, 9, nbr)
    per[1000:1400] = 0
    per[5], per[2000] = 40, 39
    bcol = np.concatenate([np.sort(rng.choice(ncb, p, replace=False)) for p in per]).astype(np.uint32)
    bval, x = random_x(rng, bcol.size * b * b, dtype), random_x(rng, ncb * b, dtype)
    A = capi.bcsr(dtype, nbr * b, ncb * b, b, b, np.concatenate([[0], np.cumsum(per)]), bcol, bval, bval.size,
                  np.full(bcol.size, b * b, np.uint32))
    row = np.repeat(np.arange(nbr), per)[:, None, None] * b + np.arange(b)[None, :, None] + np.zeros((1, 1, b), int)
    col = bcol.astype(int)[:, None, None] * b + np.arange(b)[None, None, :] + np.zeros((1, b, 1), int)
    for parts in (1, 7, 300, 2048, 5000):
        for bal in (capi.BAL_ROW, capi.BAL_BLOCK):
            plan = sp.Plan(A, sp.default_opts(nr_parts=parts, part_balance=bal))
            for _ in range(2):
                check(run(plan, x, nbr * b), nbr * b, row.reshape(-1).astype(np.uint32),
                      col.reshape(-1).astype(np.uint32), bval, x, dtype)
            if parts >= 2048:  # one or two block rows each
                assert plan.info.items > 1400 and 100 < plan.info.cta_items < 700
            plan.free()


@pytest.mark.parametrize("dtype", ["i8", "i16", "i32", "f32", "i64", "f64"])
@pytest.mark.parametrize("length", [700, 1500, 3000])
def test_long_rows_run_in_the_wide_form(dtype, length):
    lens = np.full(800, length)
    lens[::7] = 3
    want = matrix(dtype, lens)
    n = items(csr(want), want)
    limit = {1: 1024, 2: 1024, 4: 2048, 8: 10**9}[np.dtype(capi.DTYPES[dtype].np).itemsize]
    nnz = lens.sum()
    if length > limit:  # whole rows, up to 4080 nonzeros per item
        assert n <= np.ceil(800 / (4080 // length)) + 2
    else:
        assert n > nnz / 2048


@pytest.mark.parametrize("dtype", ["i8", "i32", "f32", "f64"])
@pytest.mark.parametrize("workers", [0, 8, 9, 16])
def test_many_warps_take_larger_items(dtype, workers):
    lens = np.full(20_000, 20)
    lens[5] = 30_011  # in chunks
    want = matrix(dtype, lens)
    n, nnz = items(csr(want), want, nr_workers=workers), int(lens.sum())
    assert n < nnz / 3600 if workers > 8 else n > nnz / 1500
    nrows, r, c, v, x, _ = want
    E = sp.cooe(dtype, nrows, x.size, r, c, v)
    n = items(E, want, nr_workers=workers)
    assert abs(n - nnz / (512 * max(1, workers / 4))) < 3  # 512 nonzeros for 4 warps
    for conv in ("cooe2dcsr", "cooe2bdcsr", "cooe2bdcoo"):
        items(sp.convert(conv, E, 3, 2), want, nr_workers=workers, stage_x=0)


@pytest.mark.parametrize("dtype", ["i8", "i16", "i32"])
def test_atomics_on_small_types_take_larger_items(dtype):
    want = matrix(dtype, np.full(200, 5000))
    nrows, r, c, v, x, _ = want
    E = sp.cooe(dtype, nrows, x.size, r, c, v)
    n = items(E, want, sync=capi.SYNC_ATOMIC)
    assert n == 245 if dtype != "i32" else n > 800


@pytest.mark.parametrize("b", [2, 4, 8])
def test_bcoo_lanes_by_the_items_own_block_rows(b):
    """A stripe's blocks lie in a few of its block rows: more lanes than the mean over all of them asks for."""
    rng = np.random.default_rng(b)
    n, per = 4000, 24
    r = np.repeat(np.arange(n), per)
    c = np.clip(r + rng.integers(-200, 200, r.size), 0, n - 1)
    first = np.unique(r * n + c)  # each position once
    r, c = (first // n).astype(np.uint32), (first % n).astype(np.uint32)
    v, x = random_x(rng, r.size, "f32"), random_x(rng, n, "f32")
    D = sp.convert("rbdcsr2rbdbcoo", sp.convert("cooe2rbdcsr", sp.cooe("f32", n, n, r, c, v), 4, 16), b, b)
    for o in (dict(), dict(sync=capi.SYNC_ATOMIC), dict(lanes=8)):
        plan = sp.Plan(D, sp.default_opts(**o))
        for _ in range(2):
            check(run(plan, x, n), n, r, c, v, x, "f32")
        plan.free()


@pytest.mark.parametrize("dtype,width", [("f32", 45_048), ("f64", 22_524), ("i8", 180_192)])  # 176 KB less 32 bytes
@pytest.mark.parametrize("kind", ["dbcsr", "dbcoo"])
def test_staged_x_up_to_the_limit(dtype, width, kind):
    rng = np.random.default_rng(3)
    n = 600
    for w, fits in ((width, 1), (width + 4, 0)):
        r = np.repeat(np.arange(n), 20)
        c = rng.integers(0, 2 * w, r.size)
        at = np.unique(r * (2 * w) + c)
        r, c = (at // (2 * w)).astype(np.uint32), (at % (2 * w)).astype(np.uint32)
        v, x = random_x(rng, r.size, dtype), random_x(rng, 2 * w, dtype)
        D = sp.convert("dcsr2" + kind, sp.convert("cooe2dcsr", sp.cooe(dtype, n, 2 * w, r, c, v), 1, 2), 4, 4)
        plan = sp.Plan(D, sp.default_opts(stage_x=1))
        assert plan.info.stage_x == fits
        for _ in range(2):
            check(run(plan, x, n), n, r, c, v, x, dtype)
        plan.free()
