"""Encodings and commitments whose polynomial lies inside the buffer that the
code words go to: every column is read before anything is written over it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# where the polynomial starts in the buffer of n * 4m words: its start, its
# end, odd places between, and a word before it
@pytest.mark.parametrize("place", ["start", "end", "odd", "before"])
@pytest.mark.parametrize("log_m,n", [(5, 3), (8, 5), (12, 64), (16, 20)])
def test_overlapping_polynomial(lg, ctx, log_m, n, place):
    import torch

    m = 1 << log_m
    at = {"start": 1, "end": 1 + 3 * n * m, "odd": 1 + n * m + 3, "before": 0}[place]
    poly = lg.splitmix_coeffs(log_m + n, n * m)
    want, tree, root = lg.ligero_commit(lg.to_device(poly), log_m, n, ctx)

    def buffer():
        buf = torch.zeros(4 * n * m + 4, dtype=torch.int32, device="cuda")
        words = buf[3:]  # code words from an aligned address on: word 1 of `words`
        words[at : at + n * m] = lg.to_device(poly)
        torch.cuda.synchronize()
        return words, words[at:].data_ptr(), words[1:].data_ptr()

    words, p, e = buffer()
    assert lg.lib.lg_rs_encode_cols(ctx.handle, p, log_m, n, e) == 0
    assert torch.equal(words[1:], want)
    words, p, e = buffer()
    t2, r2 = torch.empty_like(tree), np.zeros(32, np.uint8)
    assert lg.lib.lg_ligero_commit(ctx.handle, p, log_m, n, e, t2.data_ptr(), r2.ctypes.data) == 0
    assert torch.equal(words[1:], want) and torch.equal(t2, tree) and r2.tobytes() == root
