"""Grading without plane outputs walks a reduced netlist (constants and nets
that no surviving mark depends on left out) and may stop before the last
level.  CPU: the reduction's claims against the oracle's planes.  GPU: first
ids, counts and flags against the oracle wherever the reduction or the early
stop can go wrong."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import circuits
import helpers

P = helpers.pdf()
O = helpers.oracle()
SUITE = circuits.small_suite() + [("unknown", circuits.unknown_types()), ("hub", circuits.hub(200)),
                                  ("fmax8", circuits.random_small(4343, n_gates=900, n_pi=60, n_po=150, depth=9,
                                                                  fmax=8))]
NONE = 0xFFFFFFFF


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = tmp_path_factory.mktemp("probe") / "reduce_probe.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", f"-I{helpers.ROOT / 'include'}",
                    f"-I{helpers.PKG_DIR / 'csrc'}", str(helpers.ROOT / "tests" / "reduce_probe.cpp"), "-o", str(so)],
                   check=True)
    return C.CDLL(str(so))


def reduction(probe, nl, fixed):
    G = nl.n_gates
    val, obs, need = np.zeros(G, np.int8), np.zeros(G, np.uint8), np.zeros(G, np.uint8)
    n = probe.probe_reduce(C.byref(nl.view()), int(fixed), *(x.ctypes.data_as(C.c_void_p) for x in (val, obs, need)))
    orig, hdr, nfi, nfo = (np.zeros(n, np.uint32) for _ in range(4))
    eoff, edges, lo = np.zeros(n + 1, np.uint64), np.zeros(len(nl.edges) + 8, np.uint32), np.zeros(G + 2, np.uint32)
    levels = probe.probe_arrays(*(x.ctypes.data_as(C.c_void_p) for x in (orig, hdr, nfi, nfo, eoff, edges, lo)))
    return val, obs, need, dict(orig=orig, nfi=nfi, nfo=nfo, eoff=eoff.astype(int), edges=edges, lo=lo[:levels + 1])


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("idx", range(len(SUITE)))
def test_reduction_against_the_oracle(probe, idx, mode):
    nl = SUITE[idx][1]
    n = 300
    want = O.grade(nl, helpers.rand_codes(np.random.default_rng(idx), nl.n_pi, n), n, mark_mode=mode, want_planes=True)
    val, obs, need, r = reduction(probe, nl, mode >= 2)
    for g in range(nl.n_gates):
        if val[g] >= 0:
            assert np.all(want.sim[g] == val[g])  # S0 or S1 for every pair
        if want.mark[g].any():
            assert obs[g] and need[g]
        assert not (need[g] and val[g] >= 0)
    # the reduced netlist: needed gates in level order, the same fan-ins in
    # order (constants replaced), observable fan-outs in order
    kept = [int(g) for g in r["orig"] if g != NONE]
    assert sorted(kept) == [g for g in range(nl.n_gates) if need[g]]
    new = {g: k for k, g in enumerate(r["orig"]) if g != NONE}
    c0 = int(r["lo"][1]) - 2
    level = np.searchsorted(r["lo"], np.arange(len(r["orig"])), side="right") - 1
    assert list(r["orig"][c0:c0 + 2]) == [NONE, NONE] and r["lo"][-1] == len(r["orig"])
    for g, k in new.items():
        e = r["edges"][r["eoff"][k]:r["eoff"][k + 1]]
        fin = [new[int(f)] if val[f] < 0 else c0 + int(val[f]) for f in nl.fanins(g)]
        fout = [new[int(f)] for f in nl.fanouts(g) if obs[f]] if obs[g] else []
        assert list(e) == fin + fout and r["nfi"][k] == len(fin) and r["nfo"][k] == len(fout)
        assert (level[k] == 0) == (nl.nfi[g] == 0) and all(level[f] < level[k] for f in fin)


def grade_both(nl, codes, n, mode, **opts):
    want = O.grade(nl, codes, n, mark_mode=mode)
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl, mark_mode=mode, **opts)
    s = P.State(c)
    tot = P.grade(c, s, v, t, n)
    fx, fy, total = s.snapshot()
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    assert tot.value == want.total == total.value and total.flags == want.flags
    return want


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [1, 4, 8, 32, 64, 128])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_suite_without_planes(mode, tile):
    for idx, (_, nl) in enumerate(SUITE):
        rng = np.random.default_rng(900 + idx)
        for n in (33, 2100):
            grade_both(nl, helpers.rand_codes(rng, nl.n_pi, n), n, mode, tile_words=tile)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [4, 32])
def test_inputs_over_several_pieces(tile):
    """The first pieces of inputs never transition: the walk goes on to the
    pieces that do."""
    nl = circuits.random_small(51, n_gates=6000, n_pi=4000, n_po=400, depth=10, mask=circuits.MARKING_TYPES)
    codes = helpers.rand_codes(np.random.default_rng(1), nl.n_pi, 200)
    codes[:3500] &= 1
    want = grade_both(nl, codes, 200, 0, tile_words=tile)
    assert want.total > 0
    codes[:] &= 1  # and none at all
    assert grade_both(nl, codes, 200, 0, tile_words=tile).total == 0


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [4, 32])
def test_mark_carried_past_silent_levels(tile):
    """A mark whose only carrier sits far above: levels without a mark lie
    between, and the walk must not stop at them."""
    depth = 40
    levels, types, fan = [[0, 1]], {0: P.INPT, 1: P.INPT}, {0: [], 1: []}
    for l in range(1, depth):  # a chain off input 1, which never transitions
        levels.append([l + 1])
        types[l + 1], fan[l + 1] = P.BUFF, [l]
    top = depth + 1
    levels.append([top])
    types[top], fan[top] = P.AND, [0, depth]
    nl = P.Netlist.from_fanins(levels, types, [fan[i] for i in range(top + 1)], [top])
    codes = np.array([[3, 2, 0, 3] * 30, [1] * 120], np.uint8)
    for mode in range(4):
        assert grade_both(nl, codes, 120, mode, tile_words=tile).total > 0


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [4, 32])
def test_fanout_past_16_bits(tile):
    """Above 65,535 fan-outs a record keeps no reach: the walk goes to the end."""
    nl = circuits.hub(66000)
    grade_both(nl, helpers.rand_codes(np.random.default_rng(4), nl.n_pi, 100), 100, 0, tile_words=tile)


@pytest.mark.gpu
def test_first_ids_set_by_the_caller_on_nets_that_cannot_mark():
    """Ids restored onto unobservable nets make no difference to the count."""
    nl = circuits.random_small(1002, n_gates=300, n_pi=20, n_po=40, depth=9)
    n = 500
    codes = helpers.rand_codes(np.random.default_rng(2), nl.n_pi, n)
    v, t = P.planes_from_codes(codes)
    totals = []
    for planes in (False, True):
        c = P.Circuit(nl)
        s = P.State(c)
        s.restore(np.arange(nl.n_gates) % n, np.full(nl.n_gates, NONE), P.Totals_t())
        out = [np.zeros((nl.n_gates, v.shape[1]), np.uint32) for _ in range(3)] if planes else [None] * 3
        totals.append((P.grade(c, s, v, t, n, 0, *out).value, s.snapshot()[0].tolist(), s.snapshot()[1].tolist()))
    assert totals[0] == totals[1]
