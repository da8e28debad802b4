"""Device memory of the request server: what a dropped model or survey held is free for the process's
other allocations at once, or when the last request that uses it has ended, as is everything after
close()."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20
SLACK = 48 * MB   # contexts, streams and rounding of the allocator


def free_bytes():
    import torch
    return torch.cuda.mem_get_info(0)[0]


def settles(at_least, seconds=5.0):
    end = time.time() + seconds
    while free_bytes() < at_least and time.time() < end:
        time.sleep(0.01)
    return free_bytes() >= at_least


@pytest.fixture()
def server():
    import torch
    import pfast_gb300 as pg
    torch.cuda.init()
    torch.zeros(1, device="cuda")
    srv = pg.Server(device=0, slots=2, hbm_budget_gb=40)
    yield srv
    srv.close()


def small_survey(shape):
    nz, nr, nc = shape
    src = np.array([[nr // 2, nc // 2, 0]], np.int32)
    rec = np.array([(i, i, 0) for i in range(min(nr, nc))], np.int32)
    return src, np.array([len(rec)], np.int32), rec


def test_dropped_model_is_returned(server):
    big = np.full((128, 512, 1024), 2000.0)           # 512 MB
    before = free_bytes()
    server.put_model(1, big, (10.0, 10.0, 10.0))
    assert free_bytes() <= before - 400 * MB
    server.drop_model(1)
    assert settles(before - SLACK, 0.5)
    server.put_model(2, big, (10.0, 10.0, 10.0))
    server.put_model(2, big[:1, :64], (10.0, 10.0, 10.0))   # replaced by a small one
    assert settles(before - SLACK, 0.5)


def test_dropped_survey_is_returned(server):
    n = 4 << 20
    rec = np.zeros((n, 3), np.int32)
    rec[:, 0] = np.arange(n) % 8
    before = free_bytes()
    server.put_survey3d(1, (4, 8, 16), (10.0, 10.0, 10.0), np.array([[1, 1, 1]], np.int32), np.array([n], np.int32),
                        rec, np.tile([0.0, 0.0, -1.0], (n, 1)), np.full(n, 0.1))
    assert free_bytes() <= before - 100 * MB
    server.drop_survey(1)
    assert settles(before - SLACK, 0.5)


def test_model_dropped_while_in_use_is_returned_after_the_request(server):
    import pfast_gb300 as pg
    shape = (64, 256, 512)                            # 64 MB of velocities, 192 MB and more while it runs
    big = np.full(shape, 2000.0)
    before = free_bytes()
    server.put_model(1, big, (10.0, 10.0, 10.0))
    src, srnum, rec = small_survey(shape)
    server.put_survey3d(2, shape, (10.0, 10.0, 10.0), src, srnum, rec)
    t = server.submit_forward(1, 2, precision=pg.PFAST_PLAIN_FP64)
    server.drop_model(1)
    picks, _, _ = t.result()
    assert np.isfinite(picks).all() and settles(before - SLACK)


def test_everything_is_returned_after_close():
    import torch
    import pfast_gb300 as pg
    torch.zeros(1, device="cuda")
    before = free_bytes()
    srv = pg.Server(device=0, slots=2, hbm_budget_gb=40)
    srv.put_model(1, np.full((128, 512, 1024), 2000.0), (10.0, 10.0, 10.0))
    srv.close()
    assert settles(before - SLACK, 0.5)
