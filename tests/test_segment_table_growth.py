"""The set of (net, pair) firsts cannot be grown: the call that needs the larger
one fails, and later calls do not use the one that is gone."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


def test_failed_growth_of_the_table_of_firsts():
    nl = circuits.random_small(4242, n_gates=400, n_pi=30, n_po=120, depth=10)
    few, more = 8, 4000  # (net, pair) bounds below and above what the segments can set
    codes = helpers.rand_codes(np.random.default_rng(1), nl.n_pi, more)
    c = P.Circuit(nl, mark_mode=1, seg_len=5)  # 3,690 segments: tables of 32,768 and 131,072 entries
    s = P.State(c)

    def grade(state, n):
        state.reset()
        tot = P.grade(c, state, *P.planes_from_codes(codes[:, :n]), n)
        return [tot.value, *(x.tolist() for x in state.snapshot()[:2])]

    want = {n: grade(P.State(c), n) for n in (few, more)}
    assert grade(s, few) == want[few]
    P.inject_failures(P.INJECT_DEVICE_ALLOC, 1)
    try:
        with pytest.raises(P.PdfError) as e:
            grade(s, more)
        assert e.value.status == 2
    finally:
        P.inject_failures(P.INJECT_DEVICE_ALLOC, 0)
    for n in (few, more, few):
        assert grade(s, n) == want[n]
