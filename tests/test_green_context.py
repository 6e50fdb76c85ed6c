"""Calls on a stream that has a part of the SMs (a green context): the wide
kernel's cooperative grid is sized for that part."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()
O = helpers.oracle()


@pytest.fixture(params=[8, 64])
def stream(request):
    import torch
    D = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")

    def ok(r):
        if r[0] != D.CUresult.CUDA_SUCCESS:
            pytest.skip(f"no green context here: {r[0].name}")
        return r[1] if len(r) == 2 else r[1:]

    dev = ok(D.cuDeviceGet(0))
    sms = ok(D.cuDeviceGetDevResource(dev, D.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(D.cuDevSmResourceSplitByCount(1, sms, 0, request.param))
    desc = ok(D.cuDevResourceGenerateDesc(groups[:1], 1))
    ctx = ok(D.cuGreenCtxCreate(desc, dev, D.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    st = ok(D.cuGreenCtxStreamCreate(ctx, D.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(st)
    torch.cuda.synchronize()
    D.cuStreamDestroy(st)
    D.cuGreenCtxDestroy(ctx)


@pytest.mark.parametrize("name,shape", [
    ("narrow", dict(n_gates=12000, n_pi=600, n_po=1500, depth=40, mask=circuits.MARKING_TYPES)),
    ("wide", dict(n_gates=12000, n_pi=1500, n_po=3000, depth=7, mask=circuits.MARKING_TYPES)),
])
def test_grading_on_a_part_of_the_sms(stream, name, shape):
    import torch
    nl, n = circuits.random_small(71, **shape), 3000
    codes = helpers.rand_codes(np.random.default_rng(3), nl.n_pi, n)
    want = O.grade(nl, codes, n, mark_mode=1, want_planes=True)
    v, t = P.planes_from_codes(codes)
    c = P.Circuit(nl, mark_mode=1)
    s = P.State(c)
    out = [torch.zeros((nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    for planes in ([], out):
        s.reset()
        assert P.grade(c, s, v, t, n, 0, *planes, stream=stream).value == want.total
        fx, fy, _ = s.snapshot()
        np.testing.assert_array_equal(fx, want.first_x)
        np.testing.assert_array_equal(fy, want.first_y)
    P.stage_sim(c, v, t, n, out[0], out[1], stream)
    P.stage_mark(c, out[0], out[1], out[2], n, stream)
    h = [x.cpu().numpy().view(np.uint32) for x in out]
    np.testing.assert_array_equal(P.codes_from_planes(h[0], h[1], n), want.sim)
    np.testing.assert_array_equal(P.bits_from_plane(h[2], n), want.mark)
