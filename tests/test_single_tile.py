"""Circuits made for few pairs and no tile walk single calls in column blocks of
1 or 2 words (one CTA per SM); a batch of the same circuits keeps the tile.
Single calls, planes, stage calls and a batch over one circuit, bit-exact
against the CPU oracle at the edges of the rule and past max_pairs."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


@pytest.mark.parametrize("mode,max_pairs,n", [(0, 33, 33), (1, 4736, 4736), (0, 4737, 4737), (3, 9472, 9471), (1, 9473, 9473),
                                              (2, 1000, 3001)])
def test_narrow_column_blocks(mode, max_pairs, n):
    import torch
    # more gates that can mark than the resident kernel holds, on narrow levels
    nl = circuits.random_small(77, n_gates=16000, n_pi=600, n_po=900, depth=40, fmax=5, mask=circuits.MARKING_TYPES)
    codes = helpers.rand_codes(np.random.default_rng(n), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=mode, want_planes=True)
    c = P.Circuit(nl, mark_mode=mode, max_pairs=max_pairs)
    s = P.State(c)
    tw = c.info().tile_words
    ld = -(-P.words(n) // tw) * tw
    v, t = P.planes_from_codes(codes, ld)
    dv, dt = (torch.from_numpy(x.view(np.int32)).cuda() for x in (v, t))

    def same(total):
        fx, fy, tot = s.snapshot()
        np.testing.assert_array_equal(fx, want.first_x)
        np.testing.assert_array_equal(fy, want.first_y)
        assert total == want.total == tot.value

    same(P.grade(c, s, v, t, n).value)
    b = P.Batch([(c, s, dv, dt, n, 0)])
    for call in range(2):
        s.reset()
        b.run()
        same(want.total)
        s.reset()
        out = torch.full((3, nl.n_gates, ld), -1, dtype=torch.int32, device="cuda")
        same(P.grade(c, s, dv, dt, n, 0, *out).value)
        h = out.cpu().numpy().view(np.uint32)
        np.testing.assert_array_equal(P.codes_from_planes(h[0], h[1], n), want.sim)
        np.testing.assert_array_equal(P.bits_from_plane(h[2], n), want.mark)
    s.reset()
    out.fill_(-1)
    P.stage_sim(c, dv, dt, n, out[0], out[1])
    P.stage_mark(c, out[0], out[1], out[2], n)
    P.stage_merge(c, s, out[0], out[2], n, 0)
    same(P.stage_cover(c, s, out[2], n, 0).value)
    h = out.cpu().numpy().view(np.uint32)
    np.testing.assert_array_equal(P.bits_from_plane(h[2], n), want.mark)
