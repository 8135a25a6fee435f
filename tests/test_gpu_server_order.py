"""A server with one worker takes requests in the order of their submission,
judged by when they start and end: a request's latency counts from its own
submission, so latencies by themselves say nothing about the order (they fall
where preparing the next input takes longer than a proof)."""
import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(20, 18, 20, 19), (18, 16, 17)])
def test_single_worker_starts_each_after_the_one_before(lg, ctx, sizes):
    cfgs = [lg.config_for_size(L) for L in sizes]
    polys = [lg.splitmix_coeffs(i, c.poly_len) for i, c in enumerate(cfgs)]
    srv = lg.Server(0, workers=1)
    try:
        before, after, tickets = [], [], []
        for c, p in zip(cfgs, polys):
            before.append(1e3 * time.perf_counter())
            tickets.append(srv.submit(c, p, copy_input=True))
            after.append(1e3 * time.perf_counter())
        waited = [srv.wait(t) for t in tickets]
    finally:
        srv.close()
    # the server's stamp of a submission lies between `before` and `after`
    for i in range(1, len(sizes)):
        starts, ended = after[i] + waited[i][2], before[i - 1] + waited[i - 1][1]
        assert starts >= ended, i
