"""A kernel whose wait for one of its own copies runs out: the call reports an
error, and the context works on.  The waits are given no look at all, so each
runs out although its copies do land."""
import pytest

pytestmark = pytest.mark.gpu
LG_ERR_CUDA, LG_ERR_OUT_OF_MEMORY = 4, 3


@pytest.fixture
def own(lg):
    c = lg.Context(0)
    yield c
    c.close()


# the last pass alone and after four stages in registers, in at least four tiles
# an SM (fewer go without copies); strided passes of 5 and 6 stages with bulk
# copies, whose last pass waits for none
@pytest.mark.parametrize("stages,batch", [((6,), 64 * 600), ((4, 6), 64 * 40), ((5, 6), 601), ((6, 5), 601)])
@pytest.mark.parametrize("inverse", [False, True])
def test_transform_reports_and_recovers(lg, own, stages, batch, inverse):
    import torch

    log_n, call = sum(stages), lg.ifft if inverse else lg.fft
    own.set_fft_split(stages)
    src = lg.splitmix_coeffs_device(log_n, batch << log_n, own)
    want = src.clone()
    call(want, log_n, own)
    own.set_copy_wait_limit(0)
    with pytest.raises(lg.LigeritoError) as e:
        call(src.clone(), log_n, own)
    assert e.value.status == LG_ERR_CUDA
    own.set_copy_wait_limit()
    got = src.clone()
    call(got, log_n, own)
    assert torch.equal(got, want)


@pytest.mark.parametrize("log_m,n", [(8, 5), (14, 40)])
def test_commitment_reports_and_recovers(lg, own, log_m, n):
    poly = lg.splitmix_coeffs_device(log_m, n << log_m, own)
    want = lg.ligero_commit(poly, log_m, n, own)[2]
    own.set_copy_wait_limit(0)
    with pytest.raises(lg.LigeritoError) as e:
        lg.ligero_commit(poly, log_m, n, own)
    assert e.value.status == LG_ERR_CUDA
    own.set_copy_wait_limit()
    assert lg.ligero_commit(poly, log_m, n, own)[2] == want


@pytest.mark.parametrize("on_host", [False, True])
def test_proof_reports_and_recovers(lg, own, on_host):
    cfg = lg.config_for_size(20)
    poly = lg.splitmix_coeffs(9, cfg.poly_len)
    poly = poly if on_host else lg.to_device(poly)
    want = lg.prover(cfg, poly, own).to_bytes()
    own.set_copy_wait_limit(0)
    with pytest.raises(lg.LigeritoError) as e:
        lg.prover(cfg, poly, own)
    assert e.value.status == LG_ERR_CUDA
    own.set_copy_wait_limit()
    assert lg.prover(cfg, poly, own).to_bytes() == want


def test_a_call_that_fails_otherwise_leaves_no_report_behind(lg):
    # room for the first matrix and its tree but not for the folded vector: the encoding is queued
    # (its waits run out) when the allocation is refused
    cfg = lg.config_for_size(18)
    poly = lg.splitmix_coeffs_device(1, cfg.poly_len)
    c = lg.Context(0, hbm_budget_bytes=20 << 18)
    try:
        c.set_copy_wait_limit(0)
        with pytest.raises(lg.LigeritoError) as e:
            lg.prover(cfg, poly, c)
        assert e.value.status == LG_ERR_OUT_OF_MEMORY
        c.set_copy_wait_limit()
        c.synchronize()
        d = lg.splitmix_coeffs_device(1, 1 << 12, c)
        lg.fft(d, 12, c)
    finally:
        c.close()
