"""partial_eval where few outputs are left (a cluster of blocks adds up their
terms): every number of variables, outputs from one to past the last size that
splits, more variables than one launch folds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
rng = np.random.default_rng(23)

# log_len - k = 0, 3, 8 (one block's outputs), 9, 13, 14 (the last that splits)
# and 15; k = 4..9 in one launch, 10..14 in two
CASES = [(4, 4), (5, 5), (12, 4), (13, 5), (15, 7), (16, 8), (17, 9), (18, 9), (19, 6), (21, 7), (22, 9), (23, 9),
         (24, 9), (10, 10), (14, 14), (20, 12)]


@pytest.mark.parametrize("log_len,k", CASES)
def test_matches_oracle(lg, ref, ctx, log_len, k):
    e = rng.integers(0, 2**32, size=1 << log_len, dtype=np.uint64).astype(np.uint32)
    rs = rng.integers(0, 2**32, size=k, dtype=np.uint64).astype(np.uint32)
    got = lg.to_host(lg.partial_eval(lg.to_device(e), rs, ctx))
    assert (got == ref.partial_eval(e, rs, nthreads=8)).all()
