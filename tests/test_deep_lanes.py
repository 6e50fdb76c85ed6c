"""A circuit of more levels than the thread-per-gate kernel takes pieces
(65,536), at a lane tile, which bounds them by nothing: accepted and graded,
whatever of it could be left out of the walk."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


def _deep(levels=66000, dead=8000):
    """A chain of NOT and BUFF gates beside gates of constant value."""
    G = 2 + dead + levels
    lv = [[0, 1], list(range(2, 2 + dead + 1))] + [[g] for g in range(3 + dead, G)]
    types = [P.INPT, P.INPT] + [P.XOR] * dead + [P.NOT if k % 3 == 0 else P.BUFF for k in range(levels)]
    fanins = [[], []] + [[0, 1]] * dead + [[0]] + [[g - 1] for g in range(3 + dead, G)]
    return P.Netlist.from_fanins(lv, types, fanins, [G - 1])


def test_more_levels_than_pieces():
    nl, n = _deep(), 40
    codes = helpers.rand_codes(np.random.default_rng(2), nl.n_pi, n)
    want = O.grade(nl, codes, n)
    assert want.total > 0
    c = P.Circuit(nl, tile_words=32)
    s = P.State(c)
    tot = P.grade(c, s, *P.planes_from_codes(codes), n)
    fx, fy, total = s.snapshot()
    assert tot.value == want.total == total.value
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    with pytest.raises(P.PdfError) as e:  # refused as ever
        P.Circuit(nl, tile_words=4)
    assert e.value.status == 6
