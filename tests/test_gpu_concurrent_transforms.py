"""Transforms, encodings and proofs on several contexts at once, in the passes
that hand a shared-memory buffer from one unit's reads to the next unit's bulk
copies: strided passes of 5 and 6 stages and the first pass of an encoding.
Other contexts' kernels on the same SMs delay those reads."""
import threading

import pytest

pytestmark = pytest.mark.gpu
THREADS, ROUNDS = 8, 6


def _run(lg, work):
    """work(context) on THREADS contexts at once, ROUNDS times; what it raised."""
    wrong = []

    def one(bar):
        c = None
        try:
            c = lg.Context(0)
            bar.wait()
            work(c)
        except BaseException as e:  # whatever ends a thread is a failure
            wrong.append(repr(e))
            bar.abort()
        finally:
            if c is not None:
                c.close()

    for _ in range(ROUNDS):
        bar = threading.Barrier(THREADS)
        ts = [threading.Thread(target=one, args=(bar,)) for _ in range(THREADS)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    return wrong


@pytest.mark.parametrize("stages,batch", [((5, 6), 601), ((6, 5), 601), ((5, 5, 6), 64), ((6, 6, 4), 64)])
@pytest.mark.parametrize("inverse", [False, True])
def test_transforms(lg, ctx, stages, batch, inverse):
    import torch

    log_n, call = sum(stages), lg.ifft if inverse else lg.fft
    src = lg.splitmix_coeffs_device(7, batch << log_n, ctx)
    want = src.clone()
    ctx.synchronize()
    call(want, log_n, ctx)

    def work(c):
        c.set_fft_split(stages)
        for _ in range(3):
            d = src.clone()
            torch.cuda.synchronize()
            call(d, log_n, c)
            assert torch.equal(d, want)

    assert _run(lg, work) == []


@pytest.mark.parametrize("stages,n", [((5, 6), 64), ((4, 5, 5), 64), ((5, 5, 6), 16)])
def test_encodings(lg, ctx, stages, n):
    import torch

    log_m = sum(stages)
    poly = lg.splitmix_coeffs_device(8, n << log_m, ctx)
    want = lg.encode_cols(poly, log_m, n, ctx)

    def work(c):
        c.set_fft_split(stages)
        for _ in range(3):
            assert torch.equal(lg.encode_cols(poly, log_m, n, c), want)

    assert _run(lg, work) == []


def test_proofs_with_a_strided_pass_of_five(lg, ctx):
    cfg = lg.config_for_size(21)
    poly = lg.splitmix_coeffs_device(21, cfg.poly_len, ctx)
    want = lg.prover(cfg, poly, ctx).to_bytes()

    def work(c):
        c.set_fft_split((4, 5, 6))  # the first commitment's columns
        for _ in range(2):
            assert lg.prover(cfg, poly, c).to_bytes() == want

    assert _run(lg, work) == []
