"""Accuracy of the block formats' sums, and what infinities and NaN in x give.

A lane sums a piece of up to 4 products, adds two pieces and then carries on with
what its additions round off; lanes are added in a tree.  An operation whose result
has the norm of k products errs by about 0.21 sqrt(k) units of eps times a product
(the root mean square of rounding, results being spread between powers of two), so
n products in pieces of 4 (10 / 4 k per product), pairs (1), one rounding of the
lanes' sums (1) and up to five levels of lanes (4 to 5, the pieces of a row among
them) err by 0.21 sqrt(10) = 0.66 units of eps sqrt(sum of squares) at most, for any
number of blocks; 0.75 leaves room for the sample.  Added one after the other by the
same lanes, 20 blocks make 0.98 and more."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi

pytestmark = pytest.mark.gpu


def blocks(dtype, b, per, nbr, rng):
    npt = capi.DTYPES[dtype].np
    ncb = 1000
    bcol = np.sort(rng.integers(0, ncb, (nbr, per)), axis=1)
    bval, x = rng.uniform(-1, 1, (nbr, per, b, b)).astype(npt), rng.uniform(-1, 1, ncb * b).astype(npt)
    A = capi.bcsr(dtype, nbr * b, ncb * b, b, b, np.arange(nbr + 1) * per, bcol.reshape(-1).astype(np.uint32),
                  bval.reshape(-1), bval.size, np.full(nbr * per, b * b, np.uint32))
    return A, bcol, bval, x


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("b", [4, 8])
@pytest.mark.parametrize("per", [8, 20, 24, 60, 200])
def test_error_does_not_grow_with_the_blocks(dtype, b, per):
    rng = np.random.default_rng(per)
    A, bcol, bval, x = blocks(dtype, b, per, max(400, 60_000 // per), rng)
    p = bval.astype(np.longdouble) * x.reshape(-1, b)[bcol][:, :, None, :]
    want, norm = p.sum((1, 3)).reshape(-1), np.sqrt((p * p).sum((1, 3)).reshape(-1))
    for M in (A, sp.convert("bcsr2bcoo", A)):
        e = (sp.Plan(M).run_host(x) - want) / norm / np.finfo(bval.dtype).eps
        assert float(np.sqrt((e * e).mean())) < 0.75


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("b", [2, 4, 8])
@pytest.mark.parametrize("per", [1, 5, 20, 3000])  # the last in block rows longer than a chunk
def test_infinities_and_nan(dtype, b, per):
    rng = np.random.default_rng(b)
    A, bcol, bval, x = blocks(dtype, b, per, 40, rng)
    x = x.astype(np.longdouble)
    x[[0, 7 * b, 11 * b + 1]] = np.inf
    x[13 * b] = np.nan
    x[[100 * b, 101 * b]] = [1e37, -1e37]  # large, of both signs: sums stay finite
    with np.errstate(invalid="ignore", over="ignore"):
        x = x.astype(bval.dtype)
        p = bval.astype(np.longdouble) * x.astype(np.longdouble).reshape(-1, b)[bcol][:, :, None, :]
        want = p.sum((1, 3)).reshape(-1)
    for M in (A, sp.convert("bcsr2bcoo", A)):
        y = sp.Plan(M).run_host(x)
        inf, nan = np.isinf(want), np.isnan(want)
        assert np.array_equal(np.isnan(y), nan) and np.array_equal(y[inf], want[inf].astype(y.dtype))
        assert np.isfinite(y[~inf & ~nan]).all()
