"""What the device converters refuse and how far they reach, in block rows of every
length: a column past the last one is refused wherever it lies."""
import numpy as np
import pytest

from sparsep_b200 import capi

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
