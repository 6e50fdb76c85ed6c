"""pdf_state_reserve sizes each block once, for the largest need of all the
walks that calls over that many pairs can take: it frees nothing, so it does
not wait for work that other streams have in flight (a server's workers
prepare jobs while passes run), and no such call allocates afterwards."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()

SHAPES = {
    "resident": (dict(n_gates=3000, n_pi=120, n_po=400, depth=25), 0, 0),
    "narrow": (dict(n_gates=12000, n_pi=600, n_po=1500, depth=40, mask=circuits.MARKING_TYPES), 2048, 0),
    "wide": (dict(n_gates=12000, n_pi=1500, n_po=3000, depth=7, mask=circuits.MARKING_TYPES), 0, 0),
    "lanes": (dict(n_gates=12000, n_pi=1500, n_po=3000, depth=7, mask=circuits.MARKING_TYPES), 0, 32),
}


def _circuit(name):
    shape, most, tile = SHAPES[name]
    nl = circuits.random_small(71, **shape)
    return nl, P.Circuit(nl, mark_mode=1, max_pairs=most, tile_words=tile)


def _reserve(s, n):
    P.check(P.lib().pdf_state_reserve(s.h, n), "pdf_state_reserve")


@pytest.mark.parametrize("name", list(SHAPES))
def test_reserving_does_not_wait_for_the_device(name):
    import torch
    nl, c = _circuit(name)
    n = 2048
    warm = P.State(c)
    _reserve(warm, n)
    s = P.State(c)
    stream, done = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(2_000_000_000)  # about a second
        done.record()
    _reserve(s, n)
    assert not done.query()
    torch.cuda.synchronize()


@pytest.mark.parametrize("name", list(SHAPES))
def test_calls_within_a_reservation_allocate_nothing(name):
    import torch
    nl, c = _circuit(name)
    n = 2048
    codes = helpers.rand_codes(np.random.default_rng(1), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=1, want_planes=True)
    tw = c.info().tile_words
    dv, dt = (torch.from_numpy(x.view(np.int32)).cuda()
              for x in P.planes_from_codes(codes, -(-P.words(n) // tw) * tw))
    out = [torch.zeros((nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda") for _ in range(3)]
    s = P.State(c)
    _reserve(s, n)
    P.inject_failures(P.INJECT_DEVICE_ALLOC, 1 << 20)  # every allocation of the library
    try:
        assert P.grade(c, s, dv, dt, n).value == want.total
        s.reset()
        assert P.grade(c, s, dv, dt, n, 0, *out).value == want.total
        assert P.stage_cover(c, s, out[2], n, 0).value == want.total
    finally:
        P.inject_failures(P.INJECT_DEVICE_ALLOC, 0)
    s.reset()
    P.Batch([(c, s, dv, dt, n, 0)]).run()
    fx, fy, tot = s.snapshot()
    assert tot.value == want.total
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(P.bits_from_plane(out[2].cpu().numpy().view(np.uint32), n), want.mark)
