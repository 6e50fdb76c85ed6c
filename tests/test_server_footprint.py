"""A server's admission counts each job's device memory by an upper estimate:
the jobs that are active take no more than it says."""
import numpy as np
import pytest

import circuits
import helpers

pytestmark = pytest.mark.gpu

P = helpers.pdf()

SHAPES = {
    "on chip": (dict(n_gates=8000, n_pi=400, n_po=1000, depth=30, mask=circuits.MARKING_TYPES), 4),
    "staged": (dict(n_gates=30000, n_pi=1500, n_po=4000, depth=80, mask=circuits.MARKING_TYPES), 4),
    "staged, all types": (dict(n_gates=60000, n_pi=3000, n_po=8000, depth=40), 4),
    "lanes": (dict(n_gates=40000, n_pi=4000, n_po=8000, depth=10, mask=circuits.MARKING_TYPES), 64),
}


@pytest.mark.parametrize("name", list(SHAPES))
def test_active_jobs_fit_their_estimate(name):
    import torch
    torch.cuda.synchronize()
    shape, tile = SHAPES[name]
    nl, n, jobs = circuits.random_small(17, **shape), 50000, 8
    v, t = P.gen_pairs(3, nl.n_pi, n)
    # what the server and its batches take by themselves: a small job of one batch
    srv = P.Server(mark_mode=1, batch_pairs=1024, tile_words=tile)
    small = circuits.random_small(5)
    srv.submit(small, *P.gen_pairs(4, small.n_pi, 1024), 1024)
    while srv.stats().jobs_done < 1:
        srv.step()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(jobs):
        srv.submit(nl, v, t, n)
    seen = 0
    for _ in range(20000):
        before = srv.stats()
        if before.jobs_done == jobs + 1:
            break
        taken = free0 - torch.cuda.mem_get_info()[0]
        # (workers prepare and free jobs meanwhile: counted before they allocate, until they have freed)
        counted = max(before.bytes_in_use, srv.stats().bytes_in_use)
        # blocks of more than 1 MiB come in steps of 2 MiB; the batches' own lists beside
        assert taken <= counted + jobs * (8 << 20) + (32 << 20)
        seen = max(seen, before.jobs_active)
        srv.step()
    assert srv.stats().jobs_done == jobs + 1 and seen > 0
    srv.close()
