"""FFT and Reed-Solomon passes at the edges of their dispatch, bit for bit
against the oracle: tiles of the last pass with few and many blocks, ragged
vector counts, passes of 5 and 6 stages with and without bulk copies, data
that is only word-aligned."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
rng = np.random.default_rng(11)


def rand_u32(n):
    return rng.integers(0, 2**32, size=n, dtype=np.uint64).astype(np.uint32)


def on_device(lg, v, shift):
    """v on the device, `shift` words past an aligned address."""
    d = lg.to_device(np.concatenate([np.zeros(shift, np.uint32), v]))
    return d[shift:]


# log_n 4, 5: the last pass alone (4 and 5 stages); 9 and 12: one strided pass
# of 3 and 6 stages; 16: two of 5; 12 x 640: more blocks than the device holds
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("log_n,batch", [(4, 67), (5, 33), (6, 1), (9, 65), (12, 3), (12, 640), (13, 130), (16, 5)])
def test_fft_paths(lg, ref, ctx, log_n, batch, shift):
    v = rand_u32(batch << log_n)
    tw = ref.twiddles(log_n)
    d = on_device(lg, v, shift)
    lg.fft(d, log_n, ctx)
    got, want = lg.to_host(d).reshape(batch, -1), v.reshape(batch, -1)
    for i in sorted({0, 1 % batch, batch // 2, batch - 1}):
        assert (got[i] == ref.fft(want[i], tw=tw)).all()
    lg.ifft(d, log_n, ctx)
    assert (lg.to_host(d) == v).all()


# 7: the first pass has one stage; 12: two passes of 3; 20 columns of 2^16:
# four passes; 5 and 6: no first pass of its own
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("log_m,n", [(5, 3), (6, 33), (7, 1), (7, 130), (8, 5), (9, 64), (10, 17), (11, 40), (12, 9),
                                     (13, 256), (16, 20)])
def test_encode_paths(lg, ref, ctx, log_m, n, shift):
    poly = rand_u32(n << log_m)
    enc = lg.to_host(lg.encode_cols(on_device(lg, poly, shift), log_m, n, ctx)).reshape(n, -1)
    for j in sorted({0, n // 2, n - 1}):
        v = np.zeros(4 << log_m, np.uint32)
        v[: 1 << log_m] = poly[j << log_m : (j + 1) << log_m]
        assert ref.lib().lgref_rs_encode_non_systematic(32, v.ctypes.data, 1 << log_m, 4 << log_m, 4) == 0
        assert (enc[j] == v).all()
