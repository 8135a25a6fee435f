"""partial_eval's intermediate vectors count against a context's HBM budget,
and a context that only evaluates holds no arena."""
import pytest

pytestmark = pytest.mark.gpu


def test_intermediates_count_against_the_budget(lg, ctx):
    evals = lg.splitmix_coeffs_device(3, 1 << 22, ctx)
    rs = list(range(11, 24))
    want = lg.partial_eval(evals, rs, ctx)
    # 13 variables: 2^16 words (256 KiB) lie between the first launch and the next
    small = lg.Context(0, hbm_budget_bytes=128 << 10)
    try:
        with pytest.raises(lg.LigeritoError) as e:
            lg.partial_eval(evals, rs, small)
        assert e.value.status == 3
        assert small.device_bytes_in_use == 0
        lg.partial_eval(evals, rs[:6], small)  # one launch needs none
    finally:
        small.close()
    roomy = lg.Context(0, hbm_budget_bytes=1 << 20)
    try:
        assert lg.to_host(lg.partial_eval(evals, rs, roomy)).tobytes() == lg.to_host(want).tobytes()
        assert roomy.device_bytes_in_use == 0
    finally:
        roomy.close()


def test_no_arena_for_an_evaluation(lg, ctx):
    import torch

    evals = lg.splitmix_coeffs_device(3, 1 << 20, ctx)
    lg.partial_eval(evals, [5, 6, 7], ctx)
    fresh = lg.Context(0)
    try:
        fresh.synchronize()
        free = torch.cuda.mem_get_info(0)[0]
        lg.partial_eval(evals, [5, 6, 7], fresh)
        assert free - torch.cuda.mem_get_info(0)[0] < 16 << 20
    finally:
        fresh.close()
