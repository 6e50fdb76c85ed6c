"""Plane outputs of circuits whose gates that are not constant fit on chip: the
resident kernel writes their rows and constant rows are filled in.  Codes,
marks, first ids and counts against the CPU oracle, on the device at odd
pitches and offsets (nothing outside the pairs' words touched), through host
planes, and from pdf_sim alone."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()
SENT = -1515870811  # 0xA5A5A5A5

NETS = {
    "mostly_constant": lambda: circuits.random_small(71, n_gates=9000, n_pi=500, n_po=900, depth=30),
    "unknown": lambda: circuits.random_small(72, n_gates=4000, n_pi=300, n_po=500, depth=12, fmax=8,
                                             mask=circuits.WITH_FROM_DFF),
    "all_switch": lambda: circuits.random_small(73, n_gates=2500, n_pi=200, n_po=300, depth=14, fmax=7,
                                                mask=circuits.MARKING_TYPES),
    "wide_levels": lambda: circuits.random_small(74, n_gates=6400, n_pi=400, n_po=900, depth=4,
                                                 mask=circuits.MARKING_TYPES),
    "hub": lambda: circuits.hub(150),
}


def _device(rows, ld, off):
    import torch
    buf = torch.full((rows * ld + 8,), SENT, dtype=torch.int32, device="cuda")
    return buf, buf[off:off + rows * ld].view(rows, ld)


def _check(outs, want, W, n, off, ld, rows, sim_only=False):
    h = [o.cpu().numpy().view(np.uint32) for _, o in outs]
    np.testing.assert_array_equal(P.codes_from_planes(h[0][:, :W], h[1][:, :W], n), want.sim)
    if not sim_only:
        np.testing.assert_array_equal(P.bits_from_plane(h[2][:, :W], n), want.mark)
    if n % 32:
        assert not any(np.any(x[:, W - 1] >> np.uint32(n % 32)) for x in h)  # no bit past the last pair
    for (buf, _), x in zip(outs, h):
        b = buf.cpu().numpy().view(np.uint32)
        assert np.all(x[:, W:] == 0xA5A5A5A5) and np.all(b[:off] == 0xA5A5A5A5)
        assert np.all(b[off + rows * ld:] == 0xA5A5A5A5)


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("n,extra,off", [(1, 0, 0), (31, 2, 1), (128, 0, 0), (1025, 3, 2), (5000, 1, 0), (40001, 0, 0)])
@pytest.mark.parametrize("name", list(NETS))
def test_planes(name, n, extra, off, mode):
    import torch
    nl = NETS[name]()
    if n > 5000 and name != "hub" and mode != 1:
        n = 9001
    codes = helpers.rand_codes(np.random.default_rng(n + mode), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=mode, want_planes=True)
    W, G = P.words(n), nl.n_gates
    ld = W + extra
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl, mark_mode=mode)
    s = P.State(c)
    outs = [_device(G, ld, off) for _ in range(3)]
    tot = P.grade(c, s, v, t, n, 0, *(o for _, o in outs))
    torch.cuda.synchronize()
    _check(outs, want, W, n, off, ld, G)
    fx, fy, total = s.snapshot()
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    assert tot.value == want.total == total.value and tot.flags == want.flags
    codes_only = [_device(G, ld, off) for _ in range(2)]
    P.stage_sim(c, v, t, n, *(o for _, o in codes_only))
    _check(codes_only, want, W, n, off, ld, G, sim_only=True)


@pytest.mark.parametrize("which", ["host", "mark_only", "sim_only"])
def test_planes_through_the_workspace(which):
    nl, n, mode = NETS["mostly_constant"](), 700, 1
    codes = helpers.rand_codes(np.random.default_rng(9), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=mode, want_planes=True)
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl, mark_mode=mode)
    s = P.State(c)
    sv, st, mk = (np.zeros((nl.n_gates, v.shape[1]), np.uint32) for _ in range(3))
    kw = {"host": dict(sim_v=sv, sim_t=st, mark=mk), "mark_only": dict(mark=mk), "sim_only": dict(sim_v=sv, sim_t=st)}[which]
    tot = P.grade(c, s, v, t, n, 0, **kw)
    if which != "mark_only":
        np.testing.assert_array_equal(P.codes_from_planes(sv, st, n), want.sim)
    if which != "sim_only":
        np.testing.assert_array_equal(P.bits_from_plane(mk, n), want.mark)
    assert tot.value == want.total
