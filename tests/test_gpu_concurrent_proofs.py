"""Proofs on several contexts at once.  Other contexts' kernels on the same SMs
delay a unit's shared-memory reads in the FFT passes, and the next unit's bulk
copies must not overtake them: with only a barrier between the two, 4 to 13 of
400 proofs of 2^22 had a wrong column in their first commitment."""
import threading

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,rounds", [(18, 6), (22, 25)])
def test_concurrent_proofs_equal_the_single_one(lg, ctx, L, rounds):
    cfg = lg.config_for_size(L)
    poly = lg.splitmix_coeffs_device(5, cfg.poly_len, ctx)
    want, bad = lg.prover(cfg, poly, ctx).to_bytes(), []

    def work(c, bar):
        bar.wait()
        for _ in range(2):
            try:
                if lg.prover(cfg, poly, c).to_bytes() != want:
                    bad.append("bytes")
            except lg.LigeritoError as e:
                bad.append(str(e))

    for _ in range(rounds):
        ctxs, bar = [lg.Context(0) for _ in range(8)], threading.Barrier(8)
        ts = [threading.Thread(target=work, args=(c, bar)) for c in ctxs]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        for c in ctxs:
            c.close()
    assert not bad
