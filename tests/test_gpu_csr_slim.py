"""Automatic CSR items (the row kernel's slim form: 8 KB of products at a time,
fewer nonzeros per item for small matrices) and the wide form that parts and
an explicit item size keep: rows at and around the items' limits, rows cut into
chunks, runs of empty rows longer than an item's rows.  Integers bit for bit, FP
within gamma_n sum|a x|."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi
from helpers import fp_bound_ok, hi_ref, random_x

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", list(capi.DTYPES))
@pytest.mark.parametrize("size", ["one", "small", "large"])
def test_csr_items(dtype, size):
    rng = np.random.default_rng(7)
    cap = 1024 if np.dtype(capi.DTYPES[dtype].np).itemsize == 8 else 2048
    lens = {"one": np.array([1]),
            "small": np.concatenate([rng.integers(0, 9, 700), [255, 256, 257, 0, 300], np.zeros(600, int), [2]]),
            "large": np.concatenate([[cap, cap + 1, cap - 1, 1, 0, 5000, 2049, 2048], np.zeros(cap, int),
                                     np.ones(cap + 3, int), rng.integers(0, 120, 30_000), [20_000, 0]])}[size]
    nrows, ncols = lens.size, 25_000
    r = np.repeat(np.arange(nrows, dtype=np.uint32), lens)
    c = rng.integers(0, ncols, r.size).astype(np.uint32)
    v, x = random_x(rng, r.size, dtype), random_x(rng, ncols, dtype)
    A = sp.csr(dtype, nrows, ncols, *sp.synth.to_csr(nrows, r, c, v))
    for o in (dict(), dict(nr_workers=1), dict(nr_workers=16), dict(sync=capi.SYNC_ATOMIC), dict(nr_parts=9),
              dict(item_nnz=4096), dict(item_nnz=2048)):
        y = sp.Plan(A, sp.default_opts(**o)).run_host(x)
        if np.dtype(capi.DTYPES[dtype].np).kind == "f":
            ok, err, bound = fp_bound_ok(y, *hi_ref(r, c, v, x, nrows), dtype)
            assert ok, (o, float((err / bound).max()))
        else:
            want = np.zeros(nrows, np.uint64)
            np.add.at(want, r, v.astype(np.int64).astype(np.uint64) * x[c].astype(np.int64).astype(np.uint64))
            assert np.array_equal(y, want.astype(capi.DTYPES[dtype].np)), o
