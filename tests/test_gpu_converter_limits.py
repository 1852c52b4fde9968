"""What the device converters refuse, how far they reach and what they keep: a column
past the last one is refused wherever it lies, block rows may be of any length, the
scratch kept between calls can be had back."""
import ctypes as C
import time

import numpy as np
import pytest

from sparsep_b200 import capi
from test_gpu_csr2bcsr_device import TORCH

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest", [40, 300, 2048, 2049, 5000])  # of a block row: both tables, and the sort
@pytest.mark.parametrize("ncols,cb", [(6000, 4), (6001, 4), (3, 4), (6000, 1)])
@pytest.mark.parametrize("where", ["long row", "short row"])
def test_column_past_the_end_is_einval(longest, ncols, cb, where):
    import torch

    rng = np.random.default_rng(longest + ncols)
    lens = np.full(41, 3)
    lens[20] = longest - 9  # rows 20 to 23 are one block row
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    good = rng.integers(0, ncols, rowptr[-1]).astype(np.int32)
    first, last = (rowptr[20], rowptr[21] - 1) if where == "long row" else (rowptr[3], rowptr[4] - 1)
    drp = torch.from_numpy(rowptr).cuda()
    for at in (first, last):
        for col in (ncols, ncols + 1, 2**32 - 1):
            colind = good.view(np.uint32).copy()
            colind[at] = col
            dci = torch.from_numpy(colind.view(np.int32)).cuda()
            with pytest.raises(capi.SparsepError) as e:
                capi.BcsrLayout(drp.data_ptr(), dci.data_ptr(), 41, ncols, int(rowptr[-1]), 4, cb)
            assert e.value.status == capi.EINVAL
    dci = torch.from_numpy(good).cuda()
    layout = capi.BcsrLayout(drp.data_ptr(), dci.data_ptr(), 41, ncols, int(rowptr[-1]), 4, cb)
    assert layout.nblocks > 0
    layout.free()


def convert_us(per, nnz=2_000_000):
    """Time of layout and fill into 4x4 blocks, block rows of `per` nonzeros at random columns."""
    import torch

    nbr = nnz // per
    nrows, ncols = 4 * nbr, 100_000
    lens = np.full(nrows, per // 4)
    lens[::4] += per % 4
    rowptr = torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)).cuda()
    nnz = nbr * per
    g = torch.Generator(device="cuda").manual_seed(per)
    colind = torch.randint(0, ncols, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    vals = torch.rand(nnz, generator=g, device="cuda")
    times = []
    for _ in range(5):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        layout = capi.BcsrLayout(rowptr.data_ptr(), colind.data_ptr(), nrows, ncols, nnz, 4, 4)
        nb = layout.nblocks
        i32 = dict(dtype=torch.int32, device="cuda")
        bp, bc, npb = torch.empty(nbr + 1, **i32), torch.empty(nb, **i32), torch.empty(nb, **i32)
        bv = torch.empty(nb * 16, device="cuda")
        layout.fill("f32", vals.data_ptr(), bp.data_ptr(), bc.data_ptr(), bv.data_ptr(), npb.data_ptr())
        torch.cuda.synchronize()
        times.append((time.perf_counter() - t0) * 1e6)
        layout.free()
    return min(times)


def test_no_length_of_a_block_row_is_out_of_line():
    """The same number of nonzeros in block rows of every length: within a factor of
    four of the longest ones, which are sorted."""
    longest = convert_us(4000)
    us = {per: convert_us(per) for per in (64, 256, 257, 500, 1000, 2000, 2048, 2049)}
    print(us, longest)
    assert max(us.values()) < 4 * longest


def test_nonzeros_up_to_the_last_index():
    """2^32 - 1 nonzeros: the last block rows end where a 32-bit index would wrap."""
    import torch

    nnz, per = 2**32 - 1, 255
    nrows = nnz // per  # exactly: 2^32 - 1 = 255 x 16,843,009
    free = torch.cuda.mem_get_info()[0]
    if free < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    rowptr = torch.arange(nrows + 1, device="cuda", dtype=torch.int64).mul_(per).to(torch.int32)  # mod 2^32
    colind = torch.zeros(nnz, dtype=torch.int32, device="cuda")
    colind[-1] = 5  # the last row has a block of its own for its last nonzero
    vals = torch.zeros(nnz, dtype=torch.int8, device="cuda")
    vals[-1], vals[-2], vals[0] = 7, 3, 9
    layout = capi.BcsrLayout(rowptr.data_ptr(), colind.data_ptr(), nrows, 8, nnz, 1, 4)
    assert layout.nblocks == nrows + 1
    i32 = dict(dtype=torch.int32, device="cuda")
    bp, bc, npb = torch.empty(nrows + 1, **i32), torch.empty(nrows + 1, **i32), torch.empty(nrows + 1, **i32)
    bv = torch.full(((nrows + 1) * 4,), 1, dtype=torch.int8, device="cuda")
    layout.fill("i8", vals.data_ptr(), bp.data_ptr(), bc.data_ptr(), bv.data_ptr(), npb.data_ptr())
    layout.free()
    assert bp[-3:].tolist() == [nrows - 2, nrows - 1, nrows + 1] and bc[-3:].tolist() == [0, 0, 1]
    # in each of the rows all nonzeros but the last row's last lie at column 0, where the last of them stays
    assert bv[:8].tolist() == [0] * 8 and bv[-8:].tolist() == [3, 0, 0, 0, 0, 7, 0, 0]
    assert npb[-2:].tolist() == [1, 1] and int(npb.sum()) == 2


def coo2csr(dtype, nnz, nrows, seed=0):
    """One conversion of a random list; the list, and (rowptr, colind, values)."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    rows = torch.randint(0, nrows, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    cols = torch.randint(0, 2**31 - 1, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    vals = torch.randint(-100, 100, (nnz,), generator=g, device="cuda").to(getattr(torch, TORCH[dtype]))
    rowptr = torch.full((nrows + 1,), -1, dtype=torch.int32, device="cuda")
    colind, out = torch.full_like(cols, -1), torch.zeros_like(vals)
    f = getattr(capi.lib(), f"sparsep_coo2csr_device_{dtype}")
    f.argtypes = [C.c_void_p] * 3 + [C.c_uint32, C.c_uint32] + [C.c_void_p] * 4
    torch.cuda.synchronize()
    capi.check(f(rows.data_ptr(), cols.data_ptr(), vals.data_ptr(), nnz, nrows, rowptr.data_ptr(), colind.data_ptr(),
                 out.data_ptr(), None), "coo2csr_device")
    return (rows, cols, vals), (rowptr, colind, out)


def free_bytes():
    import torch

    return torch.cuda.mem_get_info()[0]


def test_trim_gives_the_kept_scratch_back():
    coo2csr("f32", 8 << 20, 1 << 20)  # at least 12 bytes per nonzero of scratch, below the 512 MB that are kept
    before = free_bytes()
    capi.trim_scratch()
    assert free_bytes() - before >= 64 << 20
    kept = free_bytes()
    capi.trim_scratch()  # nothing left to give
    assert free_bytes() == kept
    (rows, cols, vals), (_, colind, out) = coo2csr("f32", 100_000, 999)  # and the pool still serves
    order = rows.argsort(stable=True)
    assert bool((colind == cols[order]).all()) and bool((out == vals[order]).all())


def coo2csr_us(nnz, nrows=1 << 20):
    import torch

    rows = torch.randint(0, nrows, (nnz,), device="cuda", dtype=torch.int32)
    vals = torch.rand(nnz, device="cuda")
    rowptr = torch.empty(nrows + 1, dtype=torch.int32, device="cuda")
    colind, out = torch.empty_like(rows), torch.empty_like(vals)
    f = capi.lib().sparsep_coo2csr_device_f32
    f.argtypes = [C.c_void_p] * 3 + [C.c_uint32, C.c_uint32] + [C.c_void_p] * 4
    times = []
    for _ in range(5):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        capi.check(f(rows.data_ptr(), rows.data_ptr(), vals.data_ptr(), nnz, nrows, rowptr.data_ptr(),
                     colind.data_ptr(), out.data_ptr(), None))
        times.append((time.perf_counter() - t0) * 1e6)
    return min(times)


def test_scratch_beyond_what_is_kept_costs_an_allocation():
    """Scratch of more than the 512 MB that are kept comes from cudaMalloc, at most
    a few milliseconds, not from a pool that maps it anew in every call."""
    us = {n: coo2csr_us(n) for n in (8 << 20, 80 << 20)}
    print(us)
    assert us[80 << 20] < 10 * us[8 << 20] + 8000
    before = free_bytes()
    capi.trim_scratch()
    assert free_bytes() - before <= 600 << 20


@pytest.mark.parametrize("dtype", ["i8", "i16", "f32", "f64"])
@pytest.mark.parametrize("nrows", [100, 9000, 1 << 20, 1 << 24])  # one to four passes
def test_scratch_per_nonzero(dtype, nrows):
    """At most 12 bytes and a value per nonzero, as the pool shows that held nothing before."""
    nnz = 8 << 20
    capi.trim_scratch()
    (rows, cols, vals), (rowptr, colind, out) = coo2csr(dtype, nnz, nrows)
    held = free_bytes()
    capi.trim_scratch()
    held = free_bytes() - held
    assert held <= nnz * (12 + vals.element_size()) + nnz // 4 + (40 << 20)  # and digit counts, a pool's granularity
    order = rows.argsort(stable=True)
    assert bool((colind == cols[order]).all()) and bool((out == vals[order]).all())


@pytest.mark.parametrize("dtype", ["i64", "f64"])
@pytest.mark.parametrize("nrows", [100, 129, 9000, 1 << 14, 1 << 20, (1 << 21) + 1, 1 << 24])
@pytest.mark.parametrize("nnz", [1, 4097, 300_001])
def test_without_room_values_of_8_bytes_go_by_index(dtype, nrows, nnz):
    L = capi.lib()
    live = L.sparsep_test_live_allocations()
    if nrows > 128:  # one pass asks for no more
        L.sparsep_test_fail_alloc(1)
    (rows, cols, vals), (rowptr, colind, out) = coo2csr(dtype, nnz, nrows, seed=nnz)
    L.sparsep_test_fail_alloc(0)
    assert L.sparsep_test_live_allocations() == live
    order = rows.argsort(stable=True)
    assert bool((colind == cols[order]).all()) and bool((out == vals[order]).all())
    want = rows.bincount(minlength=nrows).cumsum(0)
    assert rowptr[0] == 0 and bool((rowptr[1:] == want).all())


@pytest.mark.parametrize("dtype", ["i8", "f32", "f64"])
@pytest.mark.parametrize("nrows", [129, 1 << 14, (1 << 14) + 1, 1 << 20, 1 << 24])  # two to four passes
@pytest.mark.parametrize("what", ["both", "columns", "values", "crossed"])
def test_outputs_over_the_inputs(dtype, nrows, what):
    import torch

    g = torch.Generator(device="cuda").manual_seed(nrows)
    nnz = 3_000_001  # more tiles than run at once
    rows = torch.randint(0, nrows, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    cols = torch.randint(0, 2**31 - 1, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    vals = torch.randint(-100, 100, (nnz,), generator=g, device="cuda").to(getattr(torch, TORCH[dtype]))
    order = rows.argsort(stable=True)
    want_c, want_v, want_r = cols[order], vals[order], rows.bincount(minlength=nrows).cumsum(0)
    colind = cols if what in ("both", "columns") else rows if what == "crossed" else torch.empty_like(cols)
    out = vals if what in ("both", "values") else torch.empty_like(vals)
    rowptr = torch.empty(nrows + 1, dtype=torch.int32, device="cuda")
    f = getattr(capi.lib(), f"sparsep_coo2csr_device_{dtype}")
    f.argtypes = [C.c_void_p] * 3 + [C.c_uint32, C.c_uint32] + [C.c_void_p] * 4
    torch.cuda.synchronize()
    capi.check(f(rows.data_ptr(), cols.data_ptr(), vals.data_ptr(), nnz, nrows, rowptr.data_ptr(), colind.data_ptr(),
                 out.data_ptr(), None), "coo2csr_device")
    assert torch.equal(colind, want_c) and torch.equal(out, want_v)
    assert rowptr[0] == 0 and bool((rowptr[1:] == want_r).all())
