"""Empty rows between the nonzeros of COO plans: gaps of every length around a
warp and a window of 128 elements, at a window's ends, at the cuts between
warps and items, and in tiles whose rows are mostly empty.  y holds something
else before the call; every row has to be written.  Integers bit for bit, FP
within gamma_n sum|a x|."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi
from helpers import random_x
from test_gpu_elem_chunks import check

pytestmark = pytest.mark.gpu


def run(plan, x, nrows):
    import torch

    dx = torch.from_numpy(np.concatenate([x, np.zeros(64, x.dtype)])).cuda()
    dy = torch.full((nrows,), 77, dtype=dx.dtype, device="cuda")
    plan.run_device(dx.data_ptr(), dy.data_ptr())
    torch.cuda.synchronize()
    return dy.cpu().numpy()


@pytest.mark.parametrize("dtype", list(capi.DTYPES))
@pytest.mark.parametrize("step", [1, 2, 3, 31, 32, 33, 127, 128, 129, "mixed"])
def test_gaps(dtype, step):
    rng = np.random.default_rng(5)
    n = 9000 if step == "mixed" or step < 31 else 2500
    gaps = rng.choice([0, 0, 0, 1, 2, 5, 31, 32, 33, 4000], n, p=[.2, .2, .2, .1, .1, .1, .04, .03, .02, .01]) \
        if step == "mixed" else np.full(n, step)
    rows = (np.cumsum(gaps) + 3).astype(np.uint32)
    nrows, ncols = int(rows[-1]) + 45, 2003
    cols = np.sort(rng.integers(0, ncols, n)).astype(np.uint32) if step == "mixed" else \
        rng.integers(0, ncols, n).astype(np.uint32)
    cols = cols[np.lexsort((cols, rows))]
    v, x = random_x(rng, n, dtype), random_x(rng, ncols, dtype)
    A = sp.cooe(dtype, nrows, ncols, rows, cols, v)
    for o in (dict(), dict(nr_workers=16), dict(nr_parts=7, part_balance=capi.BAL_NNZ_ELEM),
              dict(nr_parts=5, part_balance=capi.BAL_ROW)):
        plan = sp.Plan(A, sp.default_opts(**o))
        check(run(plan, x, nrows), nrows, rows, cols, v, x, dtype)
        plan.free()
    for conv in ("cooe2dcoo", "cooe2rbdcoo", "cooe2bdcoo"):
        plan = sp.Plan(sp.convert(conv, A, 16, 4))
        check(run(plan, x, nrows), nrows, rows, cols, v, x, dtype)
        plan.free()
