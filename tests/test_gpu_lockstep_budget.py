"""Batches that the HBM budget stops on the way, at many points, beside good
batches of another context: the good ones stay right, and so does the context
whose batch was stopped."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_stopped_batches_disturb_nobody(lg, ctx):
    cfg, B = lg.config_for_size(16), 64
    polys = np.stack([lg.splitmix_coeffs(300 + b, cfg.poly_len) for b in range(B)])
    d = lg.to_device(polys.ravel()).view(B, -1)
    want = [p.to_bytes() for p in lg.prove_lockstep(cfg, d, ctx)]
    wrong, stopped, done = [], [], threading.Event()

    def good():
        try:
            while not done.is_set():
                if [p.to_bytes() for p in lg.prove_lockstep(cfg, d, ctx)] != want:
                    wrong.append("a good batch")
        except Exception as e:
            wrong.append(repr(e))

    t = threading.Thread(target=good)
    t.start()
    try:
        for mb in range(64, 160, 3):
            c = lg.Context(0, hbm_budget_bytes=mb << 20)
            try:
                if [p.to_bytes() for p in lg.prove_lockstep(cfg, d, c)] != want:
                    wrong.append(mb)
            except lg.LigeritoError as e:
                assert e.status == 3
                stopped.append(mb)
                assert c.device_bytes_in_use == 0
                # what fits is right afterwards
                if lg.prover(cfg, d[0], c).to_bytes() != want[0]:
                    wrong.append((mb, "after"))
            finally:
                c.close()
    finally:
        done.set()
        t.join()
    assert wrong == []
    assert stopped and len(stopped) < len(range(64, 160, 3))
