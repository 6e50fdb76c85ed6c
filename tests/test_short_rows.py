"""pdf_merge and pdf_cover over few pairs: rows of at most 32 words are taken
several to a warp.  First ids and counts against the oracle at every number of
words where the lanes per row change, ragged pair counts and row pitches, all
widths of the cover's bitmaps; and pdf_cover over few pairs of a large circuit
takes no longer than the same work did with a thread per row."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


@pytest.mark.parametrize("tile", [1, 2, 8, 32, 128])
@pytest.mark.parametrize("n", [1, 32, 33, 64, 65, 96, 127, 160, 256, 257, 511, 513, 992, 1024, 1025])
def test_merge_and_cover(n, tile):
    import torch
    nl = circuits.random_small(4242, n_gates=397, n_pi=30, n_po=120, depth=10, mask=circuits.MARKING_TYPES)
    codes = helpers.rand_codes(np.random.default_rng(n), nl.n_pi, n)
    want = O.grade(nl, codes, n, want_planes=True)
    c = P.Circuit(nl, tile_words=tile)
    W = P.words(n)
    for ld in (W, W + 3):
        # (bits past the last pair and words past the row's are set: they are not the pairs')
        sv = np.full((nl.n_gates, ld), 0xFFFFFFFF, np.uint32)
        mk = sv.copy()
        v, _ = P.planes_from_codes(want.sim)
        m, _ = P.planes_from_codes(want.mark.astype(np.uint8))
        past = np.uint32(0) if n % 32 == 0 else np.uint32(0xFFFFFFFF) << np.uint32(n % 32)
        sv[:, :W], mk[:, :W] = v, m
        mk[:, W - 1] |= past
        dv, dm = (torch.from_numpy(x.view(np.int32)).cuda() for x in (sv, mk))
        s = P.State(c)
        P.stage_merge(c, s, dv, dm, n, 0)
        tot = P.stage_cover(c, s, dm, n, 0)
        fx, fy, _ = s.snapshot()
        np.testing.assert_array_equal(fx, want.first_x)
        np.testing.assert_array_equal(fy, want.first_y)
        assert tot.value == want.total


def test_few_pairs_of_a_large_circuit():
    """The passes over the mark plane, 200,000 rows of one word: under 25 us
    (bitmap 2, merge 21 with a thread or a warp per row at first; 40 and 28 with
    a warp per row)."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    nl, n = circuits.random_small(71, n_gates=200000, n_pi=15000, n_po=15000, depth=40, mask=circuits.MARKING_TYPES), 32
    c = P.Circuit(nl, max_pairs=n)
    s = P.State(c)
    v, t = P.gen_pairs(1, nl.n_pi, n)
    out = [torch.zeros((nl.n_gates, 1), dtype=torch.int32, device="cuda") for _ in range(3)]
    P.stage_sim(c, v, t, n, out[0], out[1])
    P.stage_mark(c, *out, n)
    P.stage_merge(c, s, out[0], out[2], n, 0)
    P.stage_cover(c, s, out[2], n, 0)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        for _ in range(5):
            P.stage_merge(c, s, out[0], out[2], n, 0)
            P.stage_cover(c, s, out[2], n, 0)
        torch.cuda.synchronize()
    us = {e.key: e.device_time_total / e.count for e in p.key_averages() if "merge" in e.key or "bitmap" in e.key}
    assert len(us) == 2 and sum(us.values()) < 25
