"""What a server books for a request covers the proof's largest buffers: the
first matrix and its tree, whose size goes by the rows and not by the
coefficients."""
import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log,cols", [(22, 2), (22, 4), (24, 6)])
def test_request_books_matrix_and_tree(lg, ctx, log, cols):
    m = log - cols
    cfg = lg.ProverConfig(1, (1 << m, 1 << cols), [(1 << (m - 4), 16)], cols, [4])
    poly = lg.splitmix_coeffs_device(1, cfg.poly_len, ctx)
    srv = lg.Server(0, workers=1)
    try:
        tickets = [srv.submit(cfg, poly) for _ in range(4)]
        booked, end = 0, time.time() + 20
        while booked == 0 and time.time() < end:
            st = srv.stats()
            booked = st["in_flight_bytes"]
            if st["completed"] == len(tickets):
                break
        for t in tickets:
            srv.wait(t)
    finally:
        srv.close()
    rows = 4 << m
    assert booked >= 4 * rows * (1 << cols) + 32 * (2 * rows - 1)
