"""What sparsep_plan_info reports about the work: `items`, the parts that a caller
asked for or else the CTA items; `cta_items`, what runs; `tiles`."""
import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mats():
    rng = np.random.default_rng(0)
    n = 6000
    lens = rng.integers(1, 60, n)
    r = np.repeat(np.arange(n, dtype=np.uint32), lens)
    c = rng.integers(0, n, r.size).astype(np.uint32)
    c = c[np.lexsort((c, r))]
    v = rng.uniform(-1, 1, r.size).astype(np.float32)
    csr = sp.csr("f32", n, n, np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32), c, v)
    bcsr = sp.convert("csr2bcsr", csr, 4, 4)
    return {"csr": csr, "cooe": sp.cooe("f32", n, n, r, c, v), "bcsr": bcsr, "bcoo": sp.convert("bcsr2bcoo", bcsr),
            "bcsr3": sp.convert("csr2bcsr", csr, 3, 3)}


def info(A, **o):
    plan = sp.Plan(A, sp.default_opts(**o))
    i = plan.info
    plan.free()
    return i


@pytest.mark.parametrize("kind", ["csr", "cooe", "bcsr", "bcoo", "bcsr3"])
def test_automatic_items(mats, kind):
    i = info(mats[kind])
    assert i.items == i.cta_items > 16 and i.tiles == 1


@pytest.mark.parametrize("kind", ["csr", "cooe", "bcsr", "bcoo"])
@pytest.mark.parametrize("parts", [1, 3])
def test_parts_are_cut(mats, kind, parts):
    i = info(mats[kind], nr_parts=parts)
    assert i.items == parts and i.cta_items > 16 and i.tiles == 1


@pytest.mark.parametrize("parts", [1, 3, 64])
def test_a_part_per_cta(mats, parts):
    """Fixed lanes per row, and block sizes without chunks."""
    for i in (info(mats["csr"], nr_parts=parts, lanes=4), info(mats["bcsr3"], nr_parts=parts)):
        assert i.items == i.cta_items == parts


def test_tiles(mats):
    for conv, n in (("cooe2dcsr", 12), ("cooe2bdcsr", 12), ("cooe2dcoo", 12), ("cooe2bdcoo", 3)):  # stripes: one per column
        D = sp.convert(conv, mats["cooe"], 4, 3)
        for parts in (0, 7):
            i = info(D, nr_parts=parts)
            assert i.tiles == n and i.cta_items >= i.items > 0, conv
