"""Plans of a given number of parts, which are cut into the items of the
automatic form where their rows run through the row kernel: parts by rows and by
nonzeros with a row longer than any item (and one of exactly an item), empty
rows and parts, more parts than rows; 1D CSR and COO and 2D tiles, with and
without atomics and with the lanes per row fixed, where a part stays one CTA's.
Each plan runs twice into a y that holds something else.  Integers bit for bit,
FP within gamma_n sum|a x|."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi
from helpers import random_x
from test_gpu_elem_chunks import check
from test_gpu_elem_gaps import run

pytestmark = pytest.mark.gpu


def matrix(dtype, seed=3):
    rng = np.random.default_rng(seed)
    lens = np.concatenate([rng.integers(0, 9, 700), np.zeros(150, int), [2048, 1024, 2049, 30_011, 0, 4097],
                           rng.integers(0, 60, 300), [9000], np.zeros(9, int)])
    ncols = 3001
    r = np.repeat(np.arange(lens.size, dtype=np.uint32), lens)
    c = rng.integers(0, ncols, r.size).astype(np.uint32)
    c = c[np.lexsort((c, r))]
    return lens, ncols, r, c, random_x(rng, r.size, dtype), random_x(rng, ncols, dtype)


def both(A, opts, want, parts=None):
    plan = sp.Plan(A, sp.default_opts(**opts))
    if parts is not None:
        assert plan.info.items <= parts
    for _ in range(2):
        check(run(plan, want[4], want[0]), *want)
    plan.free()


@pytest.mark.parametrize("dtype", list(capi.DTYPES))
@pytest.mark.parametrize("parts", [1, 2, 7, 64, 2048])
def test_parts(dtype, parts):
    lens, ncols, r, c, v, x = matrix(dtype)
    nrows = lens.size
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    want = (nrows, r, c, v, x, dtype)
    csr, coo = sp.csr(dtype, nrows, ncols, rowptr, c, v), sp.cooe(dtype, nrows, ncols, r, c, v)
    for bal in (capi.BAL_ROW, capi.BAL_NNZ):
        for o in (dict(), dict(sync=capi.SYNC_ATOMIC), dict(lanes=4), dict(nr_workers=16)):
            both(csr, dict(nr_parts=parts, part_balance=bal, **o), want, parts)
    for bal in (capi.BAL_ROW, capi.BAL_NNZ, capi.BAL_NNZ_ELEM):
        for sync in (capi.SYNC_LF, capi.SYNC_ATOMIC):
            both(coo, dict(nr_parts=parts, part_balance=bal, sync=sync), want, parts)


@pytest.mark.parametrize("dtype", ["i8", "i32", "f32", "f64"])
@pytest.mark.parametrize("conv", ["cooe2dcsr", "cooe2rbdcsr", "cooe2bdcsr", "cooe2dcoo", "cooe2bdcoo"])
def test_tiles(dtype, conv):
    lens, ncols, r, c, v, x = matrix(dtype)
    want = (lens.size, r, c, v, x, dtype)
    A = sp.cooe(dtype, lens.size, ncols, r, c, v)
    for grid in ((2, 1), (3, 2), (16, 4)):
        D = sp.convert(conv, A, *grid)
        for o in (dict(), dict(sync=capi.SYNC_ATOMIC), dict(stage_x=0), dict(lanes=8) if "csr" in conv else dict()):
            for parts in (0, 5):
                both(D, dict(nr_parts=parts, **o), want)
