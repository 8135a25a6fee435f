"""A sumcheck step's last round absorbs a triple and squeezes nothing.  With few
words pending it hashes no block either, and the two warps of the transcript
must agree on that: proofs whose pending count there takes many values (it
follows the queries drawn, so it changes with the polynomial), with other
contexts' kernels on the same SMs, against the oracle."""
import threading

import pytest

pytestmark = pytest.mark.gpu


# (log of the folded vector, rounds of each step): all in one launch a step,
# and last rounds that run in fold_round's last block (2^17 and 2^18)
@pytest.mark.parametrize("log_m,ks,seeds", [(9, [1, 2], 24), (10, [3], 24), (18, [1, 1], 3)])
def test_last_round_with_few_words_pending(lg, ref, log_m, ks, seeds):
    dims, left = [], log_m
    for k in ks:
        left -= k
        dims.append((left, k))
    pc = lg.ProverConfig(len(ks), (1 << log_m, 2), [(1 << m, 1 << n) for m, n in dims], 1, list(ks))
    rc = ref.config(len(ks), log_m, 1, [m for m, _ in dims], list(ks))
    polys = [lg.splitmix_coeffs(400 + s, pc.poly_len) for s in range(seeds)]
    want, wrong = [ref.prove(rc, p, nthreads=8) for p in polys], []

    def work(i):
        c = lg.Context(0)
        try:
            for s in range(i, seeds + i):
                if lg.prover(pc, polys[s % seeds], c).to_bytes() != want[s % seeds]:
                    wrong.append(s % seeds)
        except Exception as e:  # a thread that dies must not look like one that agreed
            wrong.append(repr(e))
        finally:
            c.close()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
