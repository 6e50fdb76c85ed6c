"""A batch of circuits with wide levels takes the lane kernel only where its
CTAs fill enough of the GPU.  Results against the oracle on both sides of that
line, and no batch much slower than at the other kernel's tile."""
import time

import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("n,jobs", [(33, 1), (1024, 3), (2048 + 31, 10), (8000, 9), (8192, 12)])
def test_batches_of_wide_circuits(n, jobs, mode):
    """1 to 96 lane CTAs."""
    import torch
    nl = circuits.random_small(71, n_gates=12000, n_pi=1500, n_po=3000, depth=7, mask=circuits.MARKING_TYPES)
    c = P.Circuit(nl, mark_mode=mode, max_pairs=n)
    tw = c.info().tile_words
    items, want = [], []
    for k in range(jobs):
        codes = helpers.rand_codes(np.random.default_rng(k % 2), nl.n_pi, n)
        ld = -(-P.words(n) // tw) * tw
        if k < 2:
            want.append(O.grade(nl, codes, n, mark_mode=mode))
        v, t = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.planes_from_codes(codes, ld))
        items.append((c, P.State(c), v, t, n, 0))
    b = P.Batch(items)
    for _ in range(3):  # launched directly, captured, replayed
        for it in items:
            it[1].reset()
        b.run()
        for k, it in enumerate(items):
            fx, fy, tot = it[1].snapshot()
            np.testing.assert_array_equal(fx, want[k % 2].first_x)
            np.testing.assert_array_equal(fy, want[k % 2].first_y)
            assert tot.value == want[k % 2].total


def _seconds(calls):
    """Median of each call's time, taken in turn."""
    import torch
    for f in calls * 3:
        f()
    ts = [[] for _ in calls]
    for _ in range(15):
        for f, x in zip(calls, ts):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            f()
            torch.cuda.synchronize()
            x.append(time.perf_counter() - t0)
    return [sorted(x)[7] for x in ts]


def test_a_batch_of_one_wide_circuit_is_no_slower_than_at_its_tile():
    import torch
    nl, n = circuits.random_small(73, n_gates=60000, n_pi=4600, n_po=4600, depth=30, mask=circuits.MARKING_TYPES), 4096
    v, t = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.gen_pairs(1, nl.n_pi, n))
    bs = []
    for tile in (0, 4):
        c = P.Circuit(nl, mark_mode=1, max_pairs=n, tile_words=tile)
        bs.append(P.Batch([(c, P.State(c), v, t, n, 0)]))
    auto, four = _seconds([b.run for b in bs])
    assert auto < 1.5 * four  # (the lane kernel's 4 CTAs: 3.3 times)
