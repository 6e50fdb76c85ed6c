"""The spill cover of a single call takes as long as that of a batch of the same
pairs (they walk the same nets, on as many CTAs): it does not run beside the
tables of the pass before it, which leave an SM no L1."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()


def test_single_call_and_batch():
    import torch
    from torch.profiler import ProfilerActivity, profile
    nl, n = circuits.random_small(3, n_gates=52510, n_pi=6563, n_po=6563, depth=2, fmax=2,
                                  mask=circuits.MARKING_TYPES), 147
    c = P.Circuit(nl, mark_mode=2, max_pairs=n)
    s = P.State(c)
    v, t = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.gen_pairs(1, nl.n_pi, n, 8))
    b = P.Batch([(c, s, v, t, n, 0)], graph=False)

    def single():
        s.reset()
        return P.grade(c, s, v, t, n).value

    def batch():
        s.reset()
        b.run()
        return s.snapshot()[2].value

    assert single() == batch()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        for _ in range(3):
            single()
            batch()
        torch.cuda.synchronize()
    us = {("batch" if "batch" in e.key else "single"): e.device_time_total / e.count
          for e in p.key_averages() if "cover_spill" in e.key}
    assert min(us.values()) > 1000  # (pairs do spill)
    assert us["single"] < 1.12 * us["batch"]
