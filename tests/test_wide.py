"""GPU parity of the wide kernel (the default for levels of 1,024 gates or
more: the whole GPU on a level, a warp per gate and segment of up to 8 chunks
of 1,024 or 2,048 pairs) and of the resident kernel's sizes, bit-exact against
the CPU oracle at the edges of chunks, segments, row pitches and fan-ins."""
import numpy as np
import pytest

import circuits
import helpers
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


def wide(seed=61, mask=circuits.ALL_TYPES, fmax=4, depth=5):
    """1,200-gate levels."""
    return circuits.random_small(seed, n_gates=700 + 1200 * depth, n_pi=700, n_po=900, depth=depth, fmax=fmax, mask=mask)


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 33, 1024, 2048 + 31])
def test_modes(n, mode):
    for nl in (wide(), wide(62, circuits.MARKING_TYPES, 8), wide(63, circuits.WITH_FROM_DFF)):
        codes = helpers.rand_codes(np.random.default_rng(n + mode), nl.n_pi, n)
        assert_same(nl, codes, n, mode)
        assert_same_lean(nl, codes, n, mode)


def assert_same_lean(nl, codes, n, mode, **opts):
    want = O.grade(nl, codes, n, mark_mode=mode)
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl, mark_mode=mode, **opts)
    s = P.State(c)
    tot = P.grade(c, s, v, t, n)
    fx, fy, total = s.snapshot()
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    assert tot.value == want.total == total.value and total.flags == want.flags


@pytest.mark.parametrize("n", [2 * 2048 - 1, 2 * 2048 + 1, 9 * 2048 + 5, 20000])
def test_chunks_and_segments(n):
    nl = wide(64, circuits.MARKING_TYPES, depth=4)
    assert_same(nl, helpers.rand_codes(np.random.default_rng(n), nl.n_pi, n), n, 0)


@pytest.mark.parametrize("off", [0, 1, 2])
@pytest.mark.parametrize("extra", [0, 1, 2, 5])
def test_device_planes_of_any_pitch_in_place(extra, off):
    """Pairs and planes on the device at odd pitches and word offsets: written
    in place, nothing outside the pairs' words touched."""
    import torch
    nl, n, mode = wide(65, circuits.MARKING_TYPES, depth=3), 2300, 1
    codes = helpers.rand_codes(np.random.default_rng(extra), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=mode, want_planes=True)
    W = P.words(n)
    ld = W + extra
    v, t = P.planes_from_codes(codes, ld)

    def at(rows, fill):
        buf = torch.full((rows * ld + 8,), fill, dtype=torch.int32, device="cuda")
        return buf, buf[off:off + rows * ld].view(rows, ld)

    (bv, dv), (bt, dt) = at(nl.n_pi, 0), at(nl.n_pi, 0)
    dv.copy_(torch.from_numpy(v.view(np.int32)))
    dt.copy_(torch.from_numpy(t.view(np.int32)))
    sent = -1515870811  # 0xA5A5A5A5
    outs = [at(nl.n_gates, sent) for _ in range(3)]
    c = P.Circuit(nl, mark_mode=mode)
    s = P.State(c)
    tot = P.grade(c, s, dv, dt, n, 0, *(o for _, o in outs))
    torch.cuda.synchronize()
    h = [o.cpu().numpy().view(np.uint32) for _, o in outs]
    np.testing.assert_array_equal(P.codes_from_planes(h[0][:, :W], h[1][:, :W], n), want.sim)
    np.testing.assert_array_equal(P.bits_from_plane(h[2][:, :W], n), want.mark)
    for (buf, _), x in zip(outs, h):
        assert np.all(x[:, W:] == 0xA5A5A5A5)
        b = buf.cpu().numpy().view(np.uint32)
        assert np.all(b[:off] == 0xA5A5A5A5) and np.all(b[off + nl.n_gates * ld:] == 0xA5A5A5A5)
    assert tot.value == want.total


def test_stage_calls_equal_the_thread_kernel_on_any_planes():
    """pdf_mark of planes that no simulation made: the same marks as the
    thread-per-gate kernel (killed gates included), before and after pruning."""
    import torch
    nl, n = wide(66, circuits.ALL_TYPES, 6, 4), 2500
    W = P.words(n)
    g = torch.Generator(device="cuda").manual_seed(3)
    sv, st = (torch.randint(-2**31, 2**31, (nl.n_gates, W), dtype=torch.int32, device="cuda", generator=g)
              for _ in range(2))
    for mode in range(4):
        got = []
        for tile in (0, 4):
            c = P.Circuit(nl, mark_mode=mode, tile_words=tile)
            mk, fm = (torch.zeros((nl.n_gates, W), dtype=torch.int32, device="cuda") for _ in range(2))
            P.stage_mark(c, sv, st, mk, n)
            P.stage_mark_forward(c, sv, st, fm, n)
            torch.cuda.synchronize()
            got.append([P.bits_from_plane(x.cpu().numpy().view(np.uint32), n) for x in (mk, fm)])
        np.testing.assert_array_equal(got[0][0], got[1][0])
        np.testing.assert_array_equal(got[0][1], got[1][1])


def test_stage_calls_compose():
    import torch
    nl, n = wide(67, circuits.MARKING_TYPES, 5, 4), 3001
    codes = helpers.rand_codes(np.random.default_rng(5), nl.n_pi, n)
    want = O.grade(nl, codes, n, want_planes=True)
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl)
    s = P.State(c)
    sv, st, mk = (torch.zeros((nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda") for _ in range(3))
    P.stage_sim(c, v, t, n, sv, st)
    P.stage_mark(c, sv, st, mk, n)
    P.stage_merge(c, s, sv, mk, n, 0)
    tot = P.stage_cover(c, s, mk, n, 0)
    fx, fy, total = s.snapshot()
    h = lambda x: x.cpu().numpy().view(np.uint32)
    np.testing.assert_array_equal(P.codes_from_planes(h(sv), h(st), n), want.sim)
    np.testing.assert_array_equal(P.bits_from_plane(h(mk), n), want.mark)
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    assert tot.value == want.total == total.value


@pytest.mark.parametrize("seg", [2, 4])
def test_segments(seg):
    nl, n = wide(68, circuits.MARKING_TYPES, 3, 4), 1500
    codes = helpers.rand_codes(np.random.default_rng(seg), nl.n_pi, n)
    out = []
    for tile in (0, 4):  # segments graded by the wide and by the thread-per-gate kernel
        c = P.Circuit(nl, seg_len=seg, tile_words=tile)
        s = P.State(c)
        tot = P.grade(c, s, *P.planes_from_codes(codes), n)
        out.append((tot.value, *(x.tolist() for x in s.snapshot()[:2])))
    assert out[0] == out[1] and out[0][0] > 0


@pytest.mark.parametrize("gates", [5200, 7000, 9000])
def test_largest_resident_netlists(gates):
    """Around the most gates that fit an SM's shared memory."""
    nl = circuits.random_small(70, n_gates=gates, n_pi=gates // 10, n_po=gates // 8, depth=40,
                               mask=circuits.MARKING_TYPES)
    for n in (100, 3000):
        assert_same_lean(nl, helpers.rand_codes(np.random.default_rng(n), nl.n_pi, n), n, 1)
