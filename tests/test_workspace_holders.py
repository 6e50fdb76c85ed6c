"""Blocks of a state's workspace that somebody else has the address of (a
captured graph, a live batch) stay allocated when a batch bound to the state
later needs more, also where that batch grades the same pairs in wider column
blocks than the captured call."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()

SHAPES = {
    # on chip
    "resident": (dict(n_gates=3000, n_pi=120, n_po=400, depth=25), 0),
    # too large for that, narrow levels: single calls over few pairs walk blocks of 1 word, batches 4
    "narrow": (dict(n_gates=12000, n_pi=600, n_po=1500, depth=40, mask=circuits.MARKING_TYPES), 0),
    "lanes": (dict(n_gates=12000, n_pi=1500, n_po=3000, depth=7, mask=circuits.MARKING_TYPES), 32),
}


def _circuit(name, most):
    shape, tile = SHAPES[name]
    nl = circuits.random_small(910, **shape)
    c = P.Circuit(nl, mark_mode=1, max_pairs=most, tile_words=tile)
    return nl, c, P.State(c)


def _pairs(nl, c, n, seed):
    import torch
    codes = helpers.rand_codes(np.random.default_rng(seed), nl.n_pi, n)
    tw = c.info().tile_words
    dv, dt = (torch.from_numpy(x.view(np.int32)).cuda()
              for x in P.planes_from_codes(codes, -(-P.words(n) // tw) * tw))
    return dv, dt, O.grade(nl, codes, n, mark_mode=1)


def _junk():
    """Takes device memory that has just been freed."""
    import torch
    return [torch.full((1 << k,), 0x5A5A5A5A, dtype=torch.int32, device="cuda") for k in range(12, 22) for _ in range(4)]


def _untouched(junk):
    return all(bool((x == 0x5A5A5A5A).all()) for x in junk)


def _equal(s, want):
    fx, fy, tot = s.snapshot()
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    assert tot.value == want.total


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("n,more", [(1056, 1056), (1056, 4096)])
def test_captured_call_before_a_batch_that_needs_more(name, n, more):
    import torch
    nl, c, s = _circuit(name, n)
    dv, dt, want = _pairs(nl, c, n, 1)
    P.grade(c, s, dv, dt, n)  # sizes the workspace of this walk
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    pairs = P.make_pairs(dv, dt, n)
    with torch.cuda.graph(graph, stream=stream):
        P.grade_mark_async(c, s, pairs, 0, None, stream.cuda_stream)
        P.grade_cover_async(c, s, stream.cuda_stream)
    bv, bt, bwant = _pairs(nl, c, more, 2)
    b = P.Batch([(c, s, bv, bt, more, 0)])
    torch.cuda.empty_cache()
    junk = _junk()
    for _ in range(2):
        s.reset()
        graph.replay()
        torch.cuda.synchronize()
        _equal(s, want)
        s.reset()
        b.run()
        _equal(s, bwant)
    assert _untouched(junk)


@pytest.mark.parametrize("name", list(SHAPES))
def test_two_batches_over_one_state_the_smaller_bound_first(name):
    import torch
    nl, c, s = _circuit(name, 4096)
    jobs = [_pairs(nl, c, n, n) for n in (500, 4096, 9000)]
    batches = [P.Batch([(c, s, v, t, n, 0)]) for (v, t, _), n in zip(jobs, (500, 4096, 9000))]
    torch.cuda.empty_cache()
    junk = _junk()
    for _ in range(3):  # launched directly, captured, replayed
        for b, (_, _, want) in zip(batches, jobs):
            s.reset()
            b.run()
            _equal(s, want)
    assert _untouched(junk)


@pytest.mark.parametrize("name", list(SHAPES))
def test_a_batch_bound_to_more_and_more_pairs_holds_its_last_block_only(name):
    """A rebinding gives up what only the binding before it held: the memory
    taken is that of the largest binding, not of all of them."""
    import torch
    nl, c, s = _circuit(name, 4096)
    sizes = [4096 * k for k in range(1, 13)]
    last = _pairs(nl, c, sizes[-1], 5)
    b = P.Batch([(c, s, last[0], last[1], 32, 0)])
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for n in sizes:
        b.rebind([(c, s, last[0], last[1], n, 0)])
        b.run()
    grown = free0 - torch.cuda.mem_get_info()[0]
    s2 = P.State(c)
    free1 = torch.cuda.mem_get_info()[0]
    b2 = P.Batch([(c, s2, last[0], last[1], sizes[-1], 0)])
    b2.run()
    _equal(s2, last[2])
    alone = free1 - torch.cuda.mem_get_info()[0]
    # (blocks of one size more than the last: the one bound before it)
    assert grown <= 2 * alone + (8 << 20)
