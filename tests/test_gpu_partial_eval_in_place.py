"""partial_eval of seven to nine variables into a place inside its input: the
result lies anywhere there, not only at a multiple of its own length."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,log_len", [(7, 17), (7, 18), (8, 19), (9, 20)])
@pytest.mark.parametrize("place", ["start", "second", "odd", "end"])
def test_result_inside_the_input(lg, ctx, k, log_len, place):
    import numpy as np

    m = 1 << (log_len - k)
    at = {"start": 0, "second": m, "odd": m // 2 + 77, "end": (1 << log_len) - m}[place]
    evals = lg.splitmix_coeffs_device(k, 1 << log_len, ctx)
    rs = np.arange(3, 3 + k, dtype=np.uint32) * np.uint32(0x9E3779B1)
    want = lg.to_host(lg.partial_eval(evals, rs, ctx))
    for _ in range(20):
        d = evals.clone()
        out = d[at : at + m]
        ctx.synchronize()
        lg.to_host(d[:1])  # the clone is there
        assert lg.lib.lg_partial_eval(ctx.handle, d.data_ptr(), log_len, rs.ctypes.data, k, out.data_ptr()) == 0
        assert (lg.to_host(out) == want).all()
