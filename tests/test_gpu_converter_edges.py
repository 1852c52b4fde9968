"""The device converters at the sizes where they change their way: block rows
around the two table sizes (256 and 2048 nonzeros) and beyond them, more rows
per block than a warp has lanes, blocks that fit shared memory or don't and
positions that repeat inside and across groups of 32; sort passes of every
digit width, input lists around one 4096-element tile, values of 1 to 8 bytes,
and two streams converting at once from one scratch pool.  Everything is
compared bit for bit with the host converters, so there is no tolerance."""
import ctypes as C
import threading

import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi
from test_gpu_coo2csr_device import device_coo2csr
from test_gpu_csr2bcsr_device import compare, device_bcsr
from helpers import random_x

pytestmark = pytest.mark.gpu


def csr_of(dtype, lens, ncols, span, rng):
    """Rows of the given lengths, columns from `span` different ones: span < length repeats them."""
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    nnz = int(rowptr[-1])
    colind = (rng.integers(0, span, nnz) * max(1, ncols // span) % ncols).astype(np.uint32)
    vals = random_x(rng, nnz, dtype)
    vals[rng.random(nnz) < 0.1] = 0
    return sp.csr(dtype, len(lens), ncols, rowptr, colind, vals), rowptr, colind, vals


@pytest.mark.parametrize("dtype", ["i8", "f32", "f64"])
@pytest.mark.parametrize("rb,cb", [(4, 4), (2, 2), (3, 5), (33, 4), (40, 1)])
@pytest.mark.parametrize("longest", [31, 32, 33, 128, 129, 255, 256, 257, 2047, 2048, 2049])
def test_block_rows_around_the_table_sizes(dtype, rb, cb, longest):
    rng = np.random.default_rng(longest * 64 + rb * 8 + cb)
    nbr, last = 70, 2  # the last block row is ragged
    lens = np.zeros((nbr - 1) * rb + min(last, rb), np.int64)
    for i in range(0, nbr, 3):  # the block row's nonzeros over its rows
        rows = np.arange(i * rb, min((i + 1) * rb, len(lens)))
        m = longest - (i % 2) if i < nbr - 1 else min(longest, 40)
        lens[rows] = np.bincount(rng.integers(0, len(rows), m), minlength=len(rows))
    ncols = 6007
    for span in (max(2, longest // 8), ncols):
        A, rowptr, colind, vals = csr_of(dtype, lens, ncols, span, rng)
        compare(dtype, A, *device_bcsr(dtype, len(lens), ncols, rowptr, colind, vals, rb, cb), rb, cb)


@pytest.mark.parametrize("dtype", ["i8", "i16", "f32", "f64"])
@pytest.mark.parametrize("nrows", [2, 128, 129, 1 << 14, (1 << 14) + 1, 1 << 21, (1 << 21) + 1])
@pytest.mark.parametrize("nnz", [1, 31, 4095, 4096, 4097, 40961])
def test_sort_passes_and_tiles(dtype, nrows, nnz):
    rng = np.random.default_rng(nrows + nnz)
    rows = rng.integers(0, nrows, nnz).astype(np.uint32)
    rows[nnz // 2:] = rows[nnz // 2:] % min(nrows, 3)  # heavy rows: their order must be kept
    rng.shuffle(rows)
    cols = np.arange(nnz, dtype=np.uint32) % 5003
    vals = random_x(rng, nnz, dtype)
    H = sp.convert("coo2csr", sp.coo(dtype, nrows, 5003, rows, cols, vals))
    rp, co, vo = device_coo2csr(dtype, nrows, rows, cols, vals)
    assert np.array_equal(rp, np.ctypeslib.as_array(H.s.rowptr, (nrows + 1,)))
    assert np.array_equal(co, np.ctypeslib.as_array(H.s.colind, (nnz,)))
    assert vo.tobytes() == np.ctypeslib.as_array(H.s.values, (nnz,)).tobytes()


def test_two_streams_at_once():
    import torch

    L = capi.lib()
    f = L.sparsep_coo2csr_device_f32
    f.argtypes = [C.c_void_p] * 3 + [C.c_uint32, C.c_uint32] + [C.c_void_p] * 4
    nrows, nnz, bad = 60_000, 400_000, []

    def work(seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        rows = torch.randint(0, nrows, (nnz,), generator=g, device="cuda", dtype=torch.int32)
        cols = torch.randint(0, 999, (nnz,), generator=g, device="cuda", dtype=torch.int32)
        vals = torch.rand(nnz, generator=g, device="cuda")
        order = torch.sort(rows, stable=True).indices
        rp = torch.zeros(nrows + 1, dtype=torch.int32, device="cuda")
        co, vo = torch.zeros_like(cols), torch.zeros_like(vals)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        for _ in range(10):
            co.zero_(), vo.zero_()
            torch.cuda.current_stream().synchronize()
            st = f(rows.data_ptr(), cols.data_ptr(), vals.data_ptr(), nnz, nrows, rp.data_ptr(), co.data_ptr(),
                   vo.data_ptr(), stream.cuda_stream)
            stream.synchronize()
            if st or not (torch.equal(co, cols[order]) and torch.equal(vo, vals[order])):
                bad.append((seed, st))

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
