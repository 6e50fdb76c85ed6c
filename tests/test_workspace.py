"""A state's workspace serves several walks (with planes and without, resident,
wide, lane).  A batch bound to a state, or a graph captured over a call, keeps
working when calls of another walk over the same state need more in between."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()

SHAPES = {
    # resident without planes, thread per gate with them
    "resident": (dict(n_gates=3000, n_pi=120, n_po=400, depth=25), 700, 0),
    # wide with and without planes; a batch takes the lane kernel
    "wide": (dict(n_gates=7700, n_pi=700, n_po=900, depth=5, mask=circuits.MARKING_TYPES), 2300, 0),
    "lanes": (dict(n_gates=12000, n_pi=1500, n_po=3000, depth=7, mask=circuits.MARKING_TYPES), 1300, 32),
}


def _job(name):
    import torch
    shape, n, tile = SHAPES[name]
    nl = circuits.random_small(900, **shape)
    c = P.Circuit(nl, mark_mode=1, tile_words=tile)
    codes = helpers.rand_codes(np.random.default_rng(n), nl.n_pi, n)
    tw = c.info().tile_words
    v, t = P.planes_from_codes(codes, -(-P.words(n) // tw) * tw)
    dv, dt = (torch.from_numpy(x.view(np.int32)).cuda() for x in (v, t))
    return nl, codes, n, c, P.State(c), v, t, dv, dt


def _others(nl, c, s, v, t, n):
    """Calls that walk every gate of the same state."""
    import torch
    W = P.words(n)
    sv, st, mk = (np.zeros((nl.n_gates, v.shape[1]), np.uint32) for _ in range(3))
    P.grade(c, s, v, t, n, 0, sv, st, mk)
    mark = torch.from_numpy(np.ascontiguousarray(mk[:, :W]).view(np.int32)).cuda()
    P.stage_cover(c, s, mark, n, 0)
    junk = [torch.full((1 << 20,), -1, dtype=torch.int32, device="cuda") for _ in range(16)]
    torch.cuda.synchronize()
    return junk


def _equal(s, want):
    fx, fy, tot = s.snapshot()
    np.testing.assert_array_equal(fx, want.first_x)
    np.testing.assert_array_equal(fy, want.first_y)
    assert tot.value == want.total


@pytest.mark.parametrize("name", list(SHAPES))
def test_batch_after_calls_of_another_walk(name):
    nl, codes, n, c, s, v, t, dv, dt = _job(name)
    want = O.grade(nl, codes, n, mark_mode=1)
    b = P.Batch([(c, s, dv, dt, n, 0)])
    for _ in range(3):  # launched directly, captured, replayed
        junk = _others(nl, c, s, v, t, n)
        s.reset()
        b.run()
        _equal(s, want)
        del junk


@pytest.mark.parametrize("name", list(SHAPES))
def test_captured_call_after_calls_of_another_walk(name):
    import torch
    nl, codes, n, c, s, v, t, dv, dt = _job(name)
    want = O.grade(nl, codes, n, mark_mode=1)
    P.grade(c, s, dv, dt, n)  # sizes the workspace of this walk
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    pairs = P.make_pairs(dv, dt, n)
    with torch.cuda.graph(graph, stream=stream):
        P.grade_mark_async(c, s, pairs, 0, None, stream.cuda_stream)
        P.grade_cover_async(c, s, stream.cuda_stream)
    for _ in range(2):
        junk = _others(nl, c, s, v, t, n)
        s.reset()
        graph.replay()
        torch.cuda.synchronize()
        _equal(s, want)
        del junk
