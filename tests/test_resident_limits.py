"""Which walks a netlist that fits on chip takes there.  The resident kernel
walks 1 to 64 words an SM at a time: over many words, netlists with room for few
are walked by the staged kernel, in calls with planes and without, alone and in
batches.  Results against the oracle on both sides of the lines, calls within a
workspace that allocate nothing, and times."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()

# gates that stay (reduced), words an SM has room for
NETS = {1: dict(n_gates=9000, n_pi=692, n_po=692, depth=40), 2: dict(n_gates=7000, n_pi=538, n_po=538, depth=40),
        4: dict(n_gates=5300, n_pi=407, n_po=407, depth=150), 8: dict(n_gates=2500, n_pi=192, n_po=192, depth=40)}


def _net(words):
    return circuits.random_small(5, mask=circuits.MARKING_TYPES, **NETS[words])


def _equal(s, tot, want):
    fx, fy, total = s.snapshot()
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    assert tot == want.total == total.value


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("words", list(NETS))
def test_both_sides_of_the_line(words, mode):
    """2 x words x SMs words; planes near it too."""
    import torch
    nl = _net(words)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = 32 * 2 * words * sms
    for n in [line - 31, line + 1] if words <= 2 else [line // 2, line + 1]:
        codes = helpers.rand_codes(np.random.default_rng(n), nl.n_pi, n)
        want = O.grade(nl, codes, n, mark_mode=mode, want_planes=True)
        v, t = P.planes_from_codes(codes)
        c = P.Circuit(nl, mark_mode=mode, max_pairs=n)
        s = P.State(c)
        _equal(s, P.grade(c, s, v, t, n).value, want)
        out = [torch.zeros((nl.n_gates, P.words(n) + 1), dtype=torch.int32, device="cuda") for _ in range(3)]
        s.reset()
        _equal(s, P.grade(c, s, v, t, n, 0, *out).value, want)
        W = P.words(n)
        h = [x.cpu().numpy().view(np.uint32)[:, :W] for x in out]
        np.testing.assert_array_equal(P.codes_from_planes(h[0], h[1], n), want.sim)
        np.testing.assert_array_equal(P.bits_from_plane(h[2], n), want.mark)
        for x in out:
            x.zero_()
        P.stage_sim(c, v, t, n, out[0], out[1])
        h = [x.cpu().numpy().view(np.uint32)[:, :W] for x in out]
        np.testing.assert_array_equal(P.codes_from_planes(h[0], h[1], n), want.sim)


@pytest.mark.parametrize("mode", [1, 3])
@pytest.mark.parametrize("jobs", [1, 5])
def test_batches(jobs, mode):
    """One job that stays on chip; five whose larger netlists do not."""
    import torch
    n = 2 * 4096 + 77
    items, want = [], []
    for k in range(jobs):
        nl = _net([1, 2, 1, 8, 1][k])
        c = P.Circuit(nl, mark_mode=mode, max_pairs=n)
        tw = c.info().tile_words
        codes = helpers.rand_codes(np.random.default_rng(k), nl.n_pi, n)
        v, t = (torch.from_numpy(x.view(np.int32)).cuda()
                for x in P.planes_from_codes(codes, -(-P.words(n) // tw) * tw))
        items.append((c, P.State(c), v, t, n, 0))
        want.append(O.grade(nl, codes, n, mark_mode=mode))
    b = P.Batch(items)
    for _ in range(3):  # launched directly, captured, replayed
        for it in items:
            it[1].reset()
        b.run()
        for it, w in zip(items, want):
            _equal(it[1], w.total, w)


@pytest.mark.parametrize("words", [1, 4])
def test_fewer_words_within_a_workspace_allocate_nothing(words):
    """Sized by a call over many words (staged), used by calls over fewer (on chip)."""
    import torch
    nl = _net(words)
    many = 32 * 8 * words * torch.cuda.get_device_properties(0).multi_processor_count
    c = P.Circuit(nl, mark_mode=1)
    s = P.State(c)
    dv, dt = (torch.zeros((nl.n_pi, P.words(many)), dtype=torch.int32, device="cuda") for _ in range(2))
    out = [torch.zeros((nl.n_gates, P.words(many)), dtype=torch.int32, device="cuda") for _ in range(3)]
    P.grade(c, s, dv, dt, many)
    P.grade(c, s, dv, dt, many, 0, *out)
    P.inject_failures(P.INJECT_DEVICE_ALLOC, 1 << 20)
    try:
        for n in (many - 1, many // 2, many // 4 + 1, many // 4, many // 8, 4000, 32, 1):
            codes = helpers.rand_codes(np.random.default_rng(n), nl.n_pi, min(n, 4000))
            v, t = P.planes_from_codes(codes, P.words(n))
            dv[:, :P.words(n)] = torch.from_numpy(v.view(np.int32)).cuda()
            dt[:, :P.words(n)] = torch.from_numpy(t.view(np.int32)).cuda()
            s.reset()
            tot = P.grade(c, s, dv, dt, n).value
            s.reset()
            assert P.grade(c, s, dv, dt, n, 0, *out).value == tot
            if n <= 4000:
                assert tot == O.grade(nl, codes, n, mark_mode=1).total
    finally:
        P.inject_failures(P.INJECT_DEVICE_ALLOC, 0)


def _walk_us(f):
    import torch
    from torch.profiler import ProfilerActivity, profile
    f()
    f()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        for _ in range(4):
            f()
        torch.cuda.synchronize()
    return sum(e.device_time_total for e in p.key_averages()
               if any(k in e.key for k in ("k_resident", "k_forward", "k_fill"))) / 4


def test_times_of_a_netlist_that_fits_only_just():
    """5,300 gates that all switch, 150 levels, 65,536 pairs: kernels that take
    306 (all planes) and 199 us (codes), 952 and 674 on chip; a reduced netlist of
    7,182 gates, 262,144 pairs: 409 and 1,276."""
    import torch
    nl, n = circuits.random_small(5, n_gates=5300, n_pi=407, n_po=407, depth=150, mask=circuits.MARKING_TYPES), 65536
    v, t = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.gen_pairs(1, nl.n_pi, n))
    out = [torch.empty((nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda") for _ in range(3)]
    c = P.Circuit(nl)
    s = P.State(c)
    assert _walk_us(lambda: P.grade(c, s, v, t, n, 0, *out)) < 600
    assert _walk_us(lambda: P.stage_sim(c, v, t, n, out[0], out[1])) < 400
    nl, n = circuits.random_small(5, n_gates=12001, n_pi=923, n_po=923, depth=45, mask=circuits.MARKING_TYPES), 262144
    v, t = (torch.from_numpy(x.view(np.int32)).cuda() for x in P.gen_pairs(1, nl.n_pi, n))
    c = P.Circuit(nl, mark_mode=1, max_pairs=n)
    s = P.State(c)
    assert _walk_us(lambda: P.grade(c, s, v, t, n)) < 800
