"""pdf_state_first_copy takes the caller's two arrays wherever they lie: rows
of one block, apart in one allocation, in the other order, or in allocations
of their own."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()


@pytest.mark.parametrize("place", ["rows", "apart", "swapped", "allocations"])
def test_arrays_anywhere(place):
    import torch
    nl = circuits.random_small(4811, n_gates=601, n_pi=41, n_po=120, depth=7, mask=circuits.MARKING_TYPES)
    G, n = nl.n_gates, 700
    v, t = P.planes_from_codes(helpers.rand_codes(np.random.default_rng(3), nl.n_pi, n))
    c = P.Circuit(nl)
    s = P.State(c)
    P.grade(c, s, v, t, n)
    want_x, want_y, _ = s.snapshot()
    if place == "allocations":  # blocks this large are allocations of their own
        a, b = (torch.full((48 << 20,), 7, dtype=torch.int32, device="cuda") for _ in range(2))
        pairs = [(a[:G], b[:G]), (b[:G], a[:G])]
    else:
        m = torch.full((3 * G + 5,), 7, dtype=torch.int32, device="cuda")
        pairs = [{"rows": (m[:G], m[G:2 * G]), "apart": (m[1:G + 1], m[2 * G + 3:3 * G + 3]),
                  "swapped": (m[G + 2:2 * G + 2], m[:G])}[place]]
    for fx, fy in pairs:
        P.first_copy(s, fx, fy, False)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(fx.cpu().numpy().view(np.uint32), want_x)
        np.testing.assert_array_equal(fy.cpu().numpy().view(np.uint32), want_y)
        fx.fill_(11)
        fy.fill_(12)
        P.first_copy(s, fx, fy, True)
        x, y, _ = s.snapshot()
        assert np.all(x == 11) and np.all(y == 12)
        P.first_copy(s, torch.from_numpy(want_x.view(np.int32)).cuda(), torch.from_numpy(want_y.view(np.int32)).cuda(), True)
    if place != "allocations":  # nothing else was written
        assert int((m == 7).sum()) == 3 * G + 5 - 2 * G
