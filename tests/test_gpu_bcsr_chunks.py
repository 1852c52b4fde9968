"""BCSR plans of 2x2, 4x4 and 8x8 blocks, which run in staged chunks of whole
block rows: chunks cut by blocks and by block rows, block rows longer than a
chunk, empty ones, ragged last block rows and columns, lanes and warps per CTA,
parts, x off its vector alignment.  Integers bit for bit, FP within gamma_n sum|a x|."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi
from helpers import fp_bound_ok, hi_ref, random_x

pytestmark = pytest.mark.gpu


def matrix(dtype, b, seed):
    rng = np.random.default_rng(seed)
    chunk = 32768 // (b * b * np.dtype(capi.DTYPES[dtype].np).itemsize)
    nbc = min(chunk, 2048) + 60
    counts = np.concatenate([rng.integers(0, 24, 90), [0, nbc, 1, nbc - 40, 0, 0], rng.integers(0, 3, 1400), [2]])
    nbr = counts.size
    nrows, ncols = nbr * b - 1, nbc * b - (b - 1)  # both ragged
    browptr = np.zeros(nbr + 1, np.uint32)
    np.cumsum(counts, out=browptr[1:])
    bcol = np.concatenate([np.sort(rng.choice(nbc, c, replace=False)) for c in counts]).astype(np.uint32)
    bval = random_x(rng, bcol.size * b * b, dtype).reshape(-1, b, b)
    brow = np.repeat(np.arange(nbr), counts)
    bval[brow == nbr - 1, (nrows - 1) % b + 1:, :] = 0
    bval[bcol == nbc - 1, :, (ncols - 1) % b + 1:] = 0
    B = dict(nrows=nrows, ncols=ncols, rb=b, cb=b, nbr=nbr, browptr=browptr, bcolind=bcol, bval=bval)
    A = capi.bcsr(dtype, nrows, ncols, b, b, browptr, bcol, bval, int((bval != 0).sum()))
    return A, B, random_x(rng, ncols, dtype)


def check(y, B, x, dtype):
    r, c, v = sp.synth.bcsr_triplets(B)
    if np.dtype(capi.DTYPES[dtype].np).kind == "f":
        ok, err, bound = fp_bound_ok(y, *hi_ref(r, c, v, x, B["nrows"]), dtype)
        assert ok, float((err / bound).max())
    else:
        want = np.zeros(B["nrows"], np.uint64)
        np.add.at(want, r, v.astype(np.int64).astype(np.uint64) * x[c].astype(np.int64).astype(np.uint64))
        assert np.array_equal(y, want.astype(capi.DTYPES[dtype].np))


@pytest.mark.parametrize("dtype", list(capi.DTYPES))
@pytest.mark.parametrize("b", [2, 4, 8])
def test_chunks(dtype, b):
    import torch

    A, B, x = matrix(dtype, b, 5 * b)
    for o in (dict(), dict(lanes=1), dict(lanes=32, nr_workers=1), dict(nr_workers=16), dict(nr_parts=7),
              dict(nr_parts=3, part_balance=capi.BAL_BLOCK), dict(sync=capi.SYNC_ATOMIC)):
        check(sp.Plan(A, sp.default_opts(**o)).run_host(x), B, x, dtype)
    # x one element off the start of its buffer, as a caller's slice may be
    plan = sp.Plan(A)
    xd = torch.from_numpy(np.concatenate([x[:1], x])).cuda()[1:]
    yd = torch.empty(B["nrows"], dtype=xd.dtype, device="cuda")
    plan.run_device(xd.data_ptr(), yd.data_ptr(), torch.cuda.current_stream().cuda_stream)
    check(yd.cpu().numpy(), B, x, dtype)


@pytest.mark.parametrize("stage_x", [0, 1])
def test_tiles(stage_x):
    A, B, x = matrix("f32", 4, 3)
    r, c, v = sp.synth.bcsr_triplets(B)
    o = np.lexsort((c, r))
    o = o[v[o] != 0]
    D = sp.convert("cooe2dcsr", sp.cooe("f32", B["nrows"], B["ncols"], r[o], c[o], v[o]), 3, 4)
    D = sp.convert("dcsr2dbcsr", D, 4, 4)
    plan = sp.Plan(D, sp.default_opts(stage_x=stage_x))
    assert plan.info.stage_x == stage_x
    check(plan.run_host(x), B, x, "f32")
