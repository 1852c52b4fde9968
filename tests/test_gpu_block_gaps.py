"""Block rows without blocks between those of BCOO plans: gaps of one to thousands
of block rows inside a chunk and across its cuts, in shared block rows and with
parts.  y holds something else before the call; every row has to be written.
Integers bit for bit, FP within gamma_n sum|a x|."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi
from helpers import random_x
from test_gpu_elem_chunks import check
from test_gpu_elem_gaps import run

pytestmark = pytest.mark.gpu


def bcoo(dtype, b, steps, per, ncb, rng):
    """Block rows `steps` apart with `per` blocks each; (matrix, nrows, its entries)."""
    brow = np.cumsum(steps) - 1 + 3  # three block rows without blocks before the first
    nbr = int(brow[-1]) + 1 + 2000   # and 2000 after the last
    counts = np.zeros(nbr, np.int64)
    counts[brow] = per
    n = int(counts.sum())
    bcol = np.concatenate([np.sort(rng.choice(ncb, p, replace=False)) for p in per]).astype(np.uint32)
    bval = random_x(rng, n * b * b, dtype)
    nrows, ncols = nbr * b - 1, ncb * b - 1  # the last of both are ragged
    rows = np.repeat(np.repeat(brow, per)[:, None, None] * b + np.arange(b)[None, :, None], b, 2)
    cols = np.repeat(bcol.astype(np.int64)[:, None, None] * b + np.arange(b)[None, None, :], b, 1)
    inside = (rows < nrows) & (cols < ncols)
    bval = np.where(inside.reshape(-1), bval, 0).astype(bval.dtype)
    A = capi.bcsr(dtype, nrows, ncols, b, b, np.concatenate([[0], np.cumsum(counts)]), bcol, bval, n * b * b,
                  np.full(n, b * b, np.uint32))
    k = inside.reshape(-1)
    return A, nrows, ncols, (rows.reshape(-1)[k].astype(np.uint32), cols.reshape(-1)[k].astype(np.uint32), bval[k])


@pytest.mark.parametrize("dtype", ["i8", "i16", "i64", "f32", "f64"])
@pytest.mark.parametrize("b", [2, 4, 8])
@pytest.mark.parametrize("kind", ["next", "every other", "far", "mixed"])
def test_gaps(dtype, b, kind):
    rng = np.random.default_rng(b)
    n = 300 if kind != "far" else 40
    steps = {"next": np.ones(n, int), "every other": np.full(n, 2), "far": np.full(n, 3000),
             "mixed": rng.choice([1, 1, 2, 3, 33, 1500], n)}[kind]
    per = np.full(n, 40) if kind == "far" else rng.choice([1, 2, 7, 60], n)
    per[n // 2] = 200  # shared by chunks
    A, nrows, ncols, (r, c, v) = bcoo(dtype, b, steps, per, 250, rng)
    O, x = sp.convert("bcsr2bcoo", A), random_x(rng, ncols, dtype)
    for o in (dict(), dict(lanes=1), dict(nr_workers=16), dict(nr_parts=7, part_balance=capi.BAL_BLOCK),
              dict(sync=capi.SYNC_ATOMIC)):
        plan = sp.Plan(O, sp.default_opts(**o))
        for _ in range(2):
            check(run(plan, x, nrows), nrows, r, c, v, x, dtype)
        plan.free()


@pytest.mark.parametrize("b", [4, 8])
def test_gaps_are_zeroed_side_by_side(b):
    """40 block rows 20,000 rows apart: in the order of the BCSR plan, whose rows are
    all written by block rows of their own (a thread per gap took 180 times that)."""
    import torch

    rng = np.random.default_rng(1)
    A, nrows, ncols, _ = bcoo("f32", b, np.full(40, 20_000 // b), np.full(40, 40), 500, rng)
    x, y = torch.rand(ncols + 64, device="cuda"), torch.empty(nrows, device="cuda")
    us = []
    for M in (A, sp.convert("bcsr2bcoo", A)):
        plan, best = sp.Plan(M), 1e9
        for _ in range(10):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            for _ in range(5):
                plan.run_device(x.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1) / 5 * 1e3)
        us.append(best)
        plan.free()
    print(us)
    assert us[1] < 10 * us[0]
