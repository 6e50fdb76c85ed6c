"""Expired waits of the staged kernel (a thread per gate, copies staged a piece
ahead), on the calls that take it: circuits with segments, pdf_mark, netlists
too large to be kept on chip, alone and in a batch.  Each call reports
PDF_ETIMEOUT with its copies drained, and the device stays usable."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()
ETIMEOUT = 4


# A wait whose copy has landed by its one poll does not expire, and of 5 blocks
# it may be that none does: hundreds of blocks of the small circuit.
def _small():
    return circuits.random_small(4242, n_gates=400, n_pi=30, n_po=120, depth=10), 60000


def _narrow():
    """8,000 gates once reduced, 200 a level."""
    return circuits.random_small(71, n_gates=12000, n_pi=600, n_po=1500, depth=40, mask=circuits.MARKING_TYPES), 4000


def _timeout(call):
    with pytest.raises(P.PdfError) as e:
        call()
    assert e.value.status == ETIMEOUT


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("make,opts", [(_small, dict(seg_len=2)), (_narrow, {}), (_narrow, dict(tile_words=8))],
                         ids=["segments", "narrow", "narrow8"])
def test_grading_calls(make, opts, mode):
    nl, n = make()
    codes = helpers.rand_codes(np.random.default_rng(mode), nl.n_pi, n)
    v, t = P.planes_from_codes(codes)
    good = P.Circuit(nl, mark_mode=mode, **opts)
    s = P.State(good)
    tot = P.grade(good, s, v, t, n)
    want = [tot.value, *(x.tolist() for x in s.snapshot()[:2])]
    if not opts.get("seg_len"):
        assert want[0] == O.grade(nl, codes, n, mark_mode=mode).total
    c = P.Circuit(nl, mark_mode=mode, wait_polls=1, **opts)
    bad = P.State(c)
    # with ids of these pairs in the state the cover has pairs to count
    bad.restore(*s.snapshot()[:2], P.Totals_t())
    for _ in range(2):
        _timeout(lambda: P.grade(c, bad, v, t, n))
    _timeout(bad.snapshot)
    s.reset()
    tot = P.grade(good, s, v, t, n)
    assert [tot.value, *(x.tolist() for x in s.snapshot()[:2])] == want


@pytest.mark.parametrize("make", [_small, _narrow], ids=["small", "narrow"])
def test_mark_calls(make):
    import torch
    nl, n = make()
    codes = helpers.rand_codes(np.random.default_rng(5), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=1, want_planes=True)
    sv, st = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.planes_from_codes(want.sim))
    mk = torch.zeros((nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda")
    c = P.Circuit(nl, mark_mode=1, wait_polls=1)
    for call in (P.stage_mark, P.stage_mark_forward, P.stage_mark):
        _timeout(lambda: call(c, sv, st, mk, n))
    good = P.Circuit(nl, mark_mode=1)
    P.stage_mark(good, sv, st, mk, n)
    np.testing.assert_array_equal(P.bits_from_plane(mk.cpu().numpy().view(np.uint32), n), want.mark)


def test_batch():
    import torch
    nl, n = _narrow()
    codes = helpers.rand_codes(np.random.default_rng(9), nl.n_pi, n)
    v, t = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.planes_from_codes(codes, 128))
    c = P.Circuit(nl, mark_mode=1, wait_polls=1)
    s = P.State(c)
    b = P.Batch([(c, s, v, t, n, 0)])
    for _ in range(3):  # launched directly, captured, replayed
        _timeout(b.run)
    good = P.Circuit(nl, mark_mode=1)
    s = P.State(good)
    P.Batch([(good, s, v, t, n, 0)]).run()
    assert s.snapshot()[2].value == O.grade(nl, codes, n, mark_mode=1).total
