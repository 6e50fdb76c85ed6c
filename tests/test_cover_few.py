"""The cover's hand-over to the large table: counts against the oracle where the
first-detecting pairs are none, one, about one and about two per SM, on
netlists whose pairs fit the small table and whose pairs do not (some not even
the large one), through grading and stage calls, several batches of a state."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


def _hubs(chains, length):
    """One input through `chains` chains of BUFFs, an output each: a pair that
    moves the input marks every net."""
    lv, fanins, types = [[0, 1]], [[], []], [P.INPT, P.INPT]
    g = 2
    for k in range(length):
        lv.append(list(range(g, g + chains)))
        for i in range(chains):
            fanins.append([0] if k == 0 else [g - chains + i])
            types.append(P.BUFF if i % 2 else P.NOT)
        g += chains
    return P.Netlist.from_fanins(lv, types, fanins, lv[-1])


# nets a pair marks: few; more than the small table holds; more than the large one
NETS = {"few": lambda: circuits.random_small(71, n_gates=12000, n_pi=600, n_po=1500, depth=40,
                                             mask=circuits.MARKING_TYPES),
        "many": lambda: _hubs(100, 20), "spill": lambda: _hubs(100, 50)}


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("name", list(NETS))
def test_counts(name, mode):
    import torch
    nl = NETS[name]()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(5)
    c = P.Circuit(nl, mark_mode=mode, max_pairs=2048)
    s, staged = P.State(c), P.State(c)
    base, fx, fy = 0, None, None
    for n in (1, 5, sms - 1, sms, sms + 1, 2 * sms, 2 * sms + 1, 700):
        codes = rng.integers(0, 4, size=(nl.n_pi, n), dtype=np.uint8)
        want = O.grade(nl, codes, n, base, mark_mode=mode, first_x=fx, first_y=fy)
        fx, fy = want.first_x, want.first_y
        v, t = P.planes_from_codes(codes)
        assert P.grade(c, s, v, t, n, base).value == want.total
        sv, st, mk = (torch.zeros((nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda") for _ in range(3))
        P.stage_sim(c, v, t, n, sv, st)
        P.stage_mark(c, sv, st, mk, n)
        P.stage_merge(c, staged, sv, mk, n, base)
        assert P.stage_cover(c, staged, mk, n, base).value == want.total
        base += n
    for state in (s, staged):
        np.testing.assert_array_equal(state.snapshot()[0], fx)
        np.testing.assert_array_equal(state.snapshot()[1], fy)


@pytest.mark.parametrize("k", [-1, 0, 1, 2])
def test_as_many_first_detecting_pairs_as_sms(k):
    """Every pair moves an input that no pair before it moved the same way."""
    import torch
    nl = NETS["few"]()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms + k if k < 2 else 2 * sms
    codes = np.zeros((nl.n_pi, n), np.uint8)
    codes[np.arange(n) % nl.n_pi, np.arange(n)] = 2 + np.arange(n) // nl.n_pi % 2
    for mode in (0, 3):
        want = O.grade(nl, codes, n, mark_mode=mode)
        c = P.Circuit(nl, mark_mode=mode, max_pairs=1024)
        s = P.State(c)
        assert P.grade(c, s, *P.planes_from_codes(codes), n).value == want.total
        np.testing.assert_array_equal(s.snapshot()[0], want.first_x)
