"""The wide kernel's grid barrier, bounded to one poll: the call reports
PDF_ETIMEOUT, the cover queued behind it reads nothing that the walk left
unfinished (also where the state already holds ids of those pairs), and the
barrier's counters are as before for the next call."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()
ETIMEOUT = 4


def _case(n=5000):
    # wide also once reduced (1,175 gates a level), and too large for the resident kernel
    nl = circuits.random_small(71, n_gates=12000, n_pi=1500, n_po=3000, depth=7, mask=circuits.MARKING_TYPES)
    return nl, helpers.rand_codes(np.random.default_rng(7), nl.n_pi, n), n


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("planes", [False, True])
def test_expired_barrier_of_a_grading_call(mode, planes):
    nl, codes, n = _case()
    want = O.grade(nl, codes, n, mark_mode=mode)
    assert want.total > 0
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl, mark_mode=mode, wait_polls=1)
    s = P.State(c)
    out = [np.zeros((nl.n_gates, v.shape[1]), np.uint32) for _ in range(3)] if planes else []
    for _ in range(3):
        # ids of these very pairs, as after an earlier grading of them: the cover
        # then has pairs to count, whatever the walk left
        tot = P.Totals_t()
        s.restore(want.first_x, want.first_y, tot)
        with pytest.raises(P.PdfError) as e:
            P.grade(c, s, v, t, n, 0, *out)
        assert e.value.status == ETIMEOUT
    s.close()
    c.close()
    good = P.Circuit(nl, mark_mode=mode)
    s = P.State(good)
    for _ in range(2):
        s.reset()
        assert P.grade(good, s, v, t, n, 0, *out).value == want.total
    fx, fy, _ = s.snapshot()
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)


def test_expired_barrier_of_the_stage_calls():
    import torch
    nl, codes, n = _case()
    v, t = P.planes_from_codes(codes)
    sv, st, mk = (torch.zeros((nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda") for _ in range(3))
    c = P.Circuit(nl, mark_mode=1, wait_polls=1)
    for call in (lambda: P.stage_sim(c, v, t, n, sv, st), lambda: P.stage_mark(c, sv, st, mk, n),
                 lambda: P.stage_mark_forward(c, sv, st, mk, n)):
        for _ in range(2):
            with pytest.raises(P.PdfError) as e:
                call()
            assert e.value.status == ETIMEOUT
    good = P.Circuit(nl, mark_mode=1)
    P.stage_sim(good, v, t, n, sv, st)
    P.stage_mark(good, sv, st, mk, n)
    torch.cuda.synchronize()
    h = lambda x: x.cpu().numpy().view(np.uint32)
    want = O.grade(nl, codes, n, mark_mode=1, want_planes=True)
    np.testing.assert_array_equal(P.codes_from_planes(h(sv), h(st), n), want.sim)
    np.testing.assert_array_equal(P.bits_from_plane(h(mk), n), want.mark)
