"""The vector kernels of conjugate gradient and power iteration at the sizes
where a thread's 16-byte loads end inside a vector, inside the grid's last pass
or just after it, with the caller's vectors on a 16-byte boundary and one
element behind one: a few iterations against the same recurrences in numpy
(FP64).  The matrix is tridiagonal (4, -1): its condition number is below 3, an
iteration rounds a vector element about ten times, so three iterations stay
within 100 roundings (2^-53 or 2^-24) of the largest element."""
import numpy as np
import pytest
import scipy.sparse as ssp

import sparsep_b200 as sp
from sparsep_b200 import capi

pytestmark = pytest.mark.gpu
PASS = 592 * 256 * 2  # 16-byte vectors that the grid takes in one pass
SIZES = [("f64", n) for n in (1, 2, 3, 7, 511, 4099, 2 * PASS - 1, 2 * PASS, 2 * PASS + 3)] + [
    ("f32", n) for n in (1, 3, 4, 5, 1025, 4 * PASS - 1, 4 * PASS + 1)]


def system(n, dtype):
    A = ssp.diags([-1.0, 4.0, -1.0], [-1, 0, 1], shape=(n, n), format="csr") if n > 1 else ssp.csr_matrix([[4.0]])
    M = sp.csr(dtype, n, n, A.indptr.astype(np.uint32), A.indices.astype(np.uint32),
               A.data.astype(capi.DTYPES[dtype].np))
    return A, sp.Plan(M)


def vector(host, tdt, shift):
    import torch

    t = torch.zeros(len(host) + 4, dtype=tdt, device="cuda")
    v = t[shift:shift + len(host)]
    v.copy_(torch.from_numpy(host))
    return t, v


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("dtype,n", SIZES)
def test_three_iterations(dtype, n, shift):
    import torch

    tdt, eps = (torch.float64, 2.0 ** -53) if dtype == "f64" else (torch.float32, 2.0 ** -24)
    rng = np.random.default_rng(n)
    b, x = (rng.uniform(-1, 1, n).astype(capi.DTYPES[dtype].np).astype(np.float64) for _ in range(2))
    A, plan = system(n, dtype)
    tb, db = vector(b, tdt, shift)
    tx, dx = vector(x, tdt, shift)
    cg = capi.CG(plan)
    it, res = cg.solve(db.data_ptr(), dx.data_ptr(), max_iters=3, rel_tol=0.0, check_every=2)
    r = b - A @ x
    p, rr = r.copy(), r @ r
    for _ in range(it):
        q = A @ p
        pq = p @ q
        alpha = rr / pq if pq else 0.0
        x, r = x + alpha * p, r - alpha * q
        new = r @ r
        p, rr = r + (new / rr if rr else 0.0) * p, new
    assert 1 <= it <= 3
    got = dx.cpu().numpy().astype(np.float64)
    assert np.abs(got - x).max() <= 100 * eps * max(1.0, np.abs(x).max())
    assert abs(res - np.sqrt(rr / (b @ b))) <= 100 * eps
    # nothing beside the vector is written
    assert not tx[:shift].any() and not tx[shift + n:].any() and torch.equal(db.double().cpu(), torch.from_numpy(b))
    cg.free()
    # power iteration from the same vector
    p0 = rng.uniform(0.5, 1, n).astype(capi.DTYPES[dtype].np).astype(np.float64)
    tp, dp = vector(p0, tdt, shift)
    pw = capi.PowerIteration(plan)
    lam, it = pw.run(dp.data_ptr(), max_iters=2, rel_tol=0.0, check_every=2)
    p, want = p0 / np.linalg.norm(p0), 0.0
    for _ in range(it):
        q = A @ p
        want = p @ q
        p = q / np.linalg.norm(q)
    assert it == 2 and abs(lam - want) <= 100 * eps * abs(want)
    assert np.abs(dp.cpu().numpy() - p).max() <= 100 * eps * np.abs(p).max()
    assert not tp[:shift].any() and not tp[shift + n:].any()
    pw.free()
    plan.free()
