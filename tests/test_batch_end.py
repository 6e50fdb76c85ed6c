"""A batch may be destroyed before its control block's upload has run and while
its last run is in flight: its pinned staging, which the one reads and the
other writes, goes only after both."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


@pytest.mark.parametrize("runs", [0, 1, 3])
def test_destroyed_with_work_in_flight(runs):
    import torch
    nl, n = circuits.random_small(77, n_gates=3000, n_pi=120, n_po=400, depth=25), 2048
    codes = helpers.rand_codes(np.random.default_rng(1), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=1)
    c = P.Circuit(nl, mark_mode=1)
    states = [P.State(c) for _ in range(40)]
    v, t = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.planes_from_codes(codes))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)  # the runs queue behind it
        b = P.Batch([(c, s, v, t, n, 0) for s in states])
        for _ in range(runs):
            b.run_async(stream.cuda_stream)
        b.close()
        pinned = torch.full((1 << 18,), 0x5A5A5A5A, dtype=torch.int32).pin_memory()  # takes what was freed
        torch.cuda.synchronize()
        assert bool((pinned == 0x5A5A5A5A).all())
        for s in states[::13]:
            if runs:
                fx, _, tot = s.snapshot()
                # (a repeated run counts the same pairs again)
                assert tot.value == runs * want.total
                np.testing.assert_array_equal(fx, want.first_x)
        for s in states:
            s.reset()
