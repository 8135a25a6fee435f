"""The pass at the root of a plain transform, whose products with the zero
twiddles are left out, against the oracle: 1 to 5 stages, forward and inverse,
with and without bulk copies, alone and before other passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
rng = np.random.default_rng(17)


# first passes of 4 (alone, word-aligned data), 1, 2, 3, 4, 5, 5 before 4, and 4 stages
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("log_n,batch", [(4, 3), (7, 9500), (8, 4800), (9, 2400), (10, 1201), (11, 601), (15, 64), (18, 6)])
def test_root_pass(lg, ref, ctx, log_n, batch, shift):
    v = rng.integers(0, 2**32, size=batch << log_n, dtype=np.uint64).astype(np.uint32)
    tw = ref.twiddles(log_n)
    d = lg.to_device(np.concatenate([np.zeros(shift, np.uint32), v]))[shift:]
    lg.fft(d, log_n, ctx)
    got, want = lg.to_host(d).reshape(batch, -1), v.reshape(batch, -1)
    for i in sorted({0, batch // 2, batch - 1}):
        assert (got[i] == ref.fft(want[i], tw=tw)).all()
    lg.ifft(d, log_n, ctx)
    assert (lg.to_host(d) == v).all()
