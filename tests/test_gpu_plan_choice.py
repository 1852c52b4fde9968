"""The learned plan choice (autotune = 1) is of the kernels as they are: against the
committed held-out times, and against a clock."""
import json

import numpy as np
import pytest

import sparsep_b200 as sp
from sparsep_b200 import plan_selector, selector, synth

pytestmark = pytest.mark.gpu


def test_held_out_regret():
    """At most 4 % above each matrix's best in total and 3 % faster than the default
    plan: weights trained on times of earlier kernels were 5.8 % above and 1.1 % faster
    on the same held-out times."""
    z, h = np.load(plan_selector.MODEL), np.load(plan_selector.DATA / "plan_heldout.npz")
    assert json.loads(str(z["meta"]))["train_samples"] == len(np.load(plan_selector.DATA / "plan_train_db.npz")["feats"])
    ev = plan_selector.evaluate(selector.selector(dict(wb=z["wb"], mean=z["mean"], std=z["std"])).scores(h["feats"]),
                                h["times"])
    assert ev["regret_total"] <= 0.04 and ev["speedup_vs_fixed_csr"] >= 1.03, ev


def test_against_a_clock():
    """Over 12 matrices that no database holds, the learned plans take no longer than
    the default ones in total (2 % for the clock)."""
    import torch

    total = [0.0, 0.0]
    for i in range(12):
        d = synth.selector_one(77, i, rows_lo=100_000, rows_hi=1_000_000, len_lo=4, len_hi=64, max_nnz=8_000_000, k_max=1)
        n, nnz = d["n"], d["colind"].size
        A = sp.csr("f32", n, n, d["rowptr"], d["colind"], np.random.default_rng(i).uniform(-1, 1, nnz).astype(np.float32))
        x, y = torch.rand(n, device="cuda"), torch.empty(n, device="cuda")
        for k, o in enumerate((dict(), dict(autotune=1))):
            plan, best = sp.Plan(A, sp.default_opts(**o)), 1e9
            for _ in range(8):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                torch.cuda.synchronize()
                e0.record()
                for _ in range(10):
                    plan.run_device(x.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
                e1.record()
                e1.synchronize()
                best = min(best, e0.elapsed_time(e1) * 100)
            total[k] += best
            plan.free()
    print(total)
    assert total[1] <= 1.02 * total[0]
