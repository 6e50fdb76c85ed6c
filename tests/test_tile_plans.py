"""A circuit made for few pairs walks blocks of 1 or 2 words in single calls,
but takes calls over more pairs than those are for, and batches, at its tile.
Results against the oracle on both sides of the line, and no call slower than
on a circuit that was made for its pairs."""
import time

import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


def _narrow(mask=circuits.MARKING_TYPES):
    """8,200 gates once reduced (too many to keep on chip), 200 a level."""
    return circuits.random_small(71, n_gates=12000, n_pi=600, n_po=1500, depth=40, mask=mask)


def _edges():
    """Pair counts around one CTA per SM in blocks of 1 word."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return [sms * 32 - 1, sms * 32, sms * 32 + 1]


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("k", [0, 1, 2])
def test_calls_over_more_pairs_than_the_circuit_was_made_for(mode, k):
    import torch
    nl, n = _narrow(), _edges()[k]
    codes = helpers.rand_codes(np.random.default_rng(k), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=mode, want_planes=True)
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl, mark_mode=mode, max_pairs=1000)
    s = P.State(c)
    h = lambda x: x.cpu().numpy().view(np.uint32)
    assert P.grade(c, s, v, t, n).value == want.total
    fx, fy, _ = s.snapshot()
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    for ld in (P.words(n), P.words(n) + 3):
        out = [torch.zeros((nl.n_gates, ld), dtype=torch.int32, device="cuda") for _ in range(3)]
        s.reset()
        assert P.grade(c, s, v, t, n, 0, *out).value == want.total
        P.stage_mark(c, out[0], out[1], out[2], n)
        s.reset()
        P.stage_merge(c, s, out[0], out[2], n, 0)
        assert P.stage_cover(c, s, out[2], n, 0).value == want.total
        np.testing.assert_array_equal(P.bits_from_plane(h(out[2])[:, :P.words(n)], n), want.mark)
        P.stage_sim(c, v, t, n, out[0], out[1])
        np.testing.assert_array_equal(P.codes_from_planes(*(h(x)[:, :P.words(n)] for x in out[:2]), n), want.sim)


def test_segments_over_more_pairs_than_the_circuit_was_made_for():
    nl, n = circuits.random_small(4242, n_gates=400, n_pi=30, n_po=120, depth=10), _edges()[2]
    codes = helpers.rand_codes(np.random.default_rng(3), nl.n_pi, n)
    got = []
    for most in (1000, n):
        c = P.Circuit(nl, mark_mode=1, max_pairs=most, seg_len=3)
        s = P.State(c)
        tot = P.grade(c, s, *P.planes_from_codes(codes), n)
        got.append([tot.value, *(x.tolist() for x in s.snapshot()[:2])])
    assert got[0] == got[1]


def test_the_plan_at_the_tile_cannot_be_allocated():
    """The call then walks the plan there is; the next one has the other."""
    nl, n = _narrow(), _edges()[2]
    codes = helpers.rand_codes(np.random.default_rng(4), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=1)
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl, mark_mode=1, max_pairs=1000)
    s = P.State(c)
    P.inject_failures(P.INJECT_DEVICE_ALLOC, 1)
    try:
        assert P.grade(c, s, v, t, n).value == want.total
    finally:
        P.inject_failures(P.INJECT_DEVICE_ALLOC, 0)
    for _ in range(2):
        s.reset()
        assert P.grade(c, s, v, t, n).value == want.total
    np.testing.assert_array_equal(s.snapshot()[0], want.first_x)


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


def test_no_slower_than_a_circuit_made_for_them():
    import torch
    nl, n = circuits.random_small(72, n_gates=20000, n_pi=1500, n_po=1500, depth=60, mask=circuits.MARKING_TYPES), 32768
    sv, st = (torch.empty((nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda") for _ in range(2))
    v, t = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.gen_pairs(1, nl.n_pi, n))
    cs = [P.Circuit(nl, max_pairs=most) for most in (1000, n)]
    over, made = _seconds([lambda c=c: P.stage_sim(c, v, t, n, sv, st) for c in cs])
    assert over < 1.5 * made  # (blocks of 1 word: 2.8 times)
