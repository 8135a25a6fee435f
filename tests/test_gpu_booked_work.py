"""The products that kernels book for their rooflines are those they execute."""
import pytest

pytestmark = pytest.mark.gpu


def _booked(ctx, call):
    ctx.set_kernel_timing(True)
    ctx.reset_kernel_stats()
    try:
        call()
        return ctx.kernel_stats(), ctx.kernel_work(), ctx.kernel_general_mults()
    finally:
        ctx.set_kernel_timing(False)
        ctx.reset_kernel_stats()


@pytest.mark.parametrize("log,batch", [(12, 640), (20, 4), (16, 33)])
@pytest.mark.parametrize("inverse", [False, True])
def test_transform_products(lg, ctx, log, batch, inverse):
    # a product a butterfly, but those of each stage's first node in the
    # root pass (twiddle zero): half of its first stage's words, a quarter of
    # the second's, ..
    d = lg.splitmix_coeffs_device(1, batch << log, ctx)
    stats, work, general = _booked(ctx, lambda: (lg.ifft if inverse else lg.fft)(d, log, ctx))
    stages = {k: int(k.split("_K")[1].split("_")[0]) for k in stats if "_K" in k}
    assert sum(stats[k][0] * K for k, K in stages.items()) == log
    words = batch << log
    skipped = words / 2 * log - sum(work[k][1] for k in stages)
    assert not any(general[k] for k in stages)
    assert skipped in [words * (1 - 2.0**-K) for K in stages.values()]


@pytest.mark.parametrize("log_m,n", [(14, 64), (12, 9)])
def test_encode_first_pass_products(lg, ctx, log_m, n):
    # a pencil of the first pass: the scaling, the first stage with two roots
    # for all quarters, and the other stages' butterflies but quarter 0's with
    # the first node
    d = lg.splitmix_coeffs_device(1, n << log_m, ctx)
    _, work, general = _booked(ctx, lambda: lg.encode_cols(d, log_m, n, ctx))
    (name,) = [k for k in work if k.endswith("_rs")]
    K = int(name.split("_K")[1].split("_")[0])
    R = 1 << K
    table = R + 4 * (K - 1) * R // 2 - (R // 2 - 1)
    assert K != 4 or table == 105
    assert work[name][1] == (n << log_m) / R * (R + table)
    assert general[name] == n << log_m  # the scaling


def test_cluster_steps_are_booked_apart(lg, ctx):
    # folded vectors of 2^14 and 2^12, a launch each
    cfg = lg.ProverConfig(2, (1 << 14, 1 << 6), [(1 << 12, 4), (1 << 10, 4)], 6, [2, 2])
    poly = lg.splitmix_coeffs_device(2, cfg.poly_len, ctx)
    stats, work, general = _booked(ctx, lambda: lg.prover(cfg, poly, ctx))
    assert stats["fold_round"][0] == 2 and "fold_round_grid" not in stats
    # an opening triple is 3 products a pair of words, the second step's glue
    # one a word, a round 4 by the table and 3 others for four words
    steps = [(1 << 14, 0), (1 << 12, 1)]
    assert work["fold_round"][1] == sum(1.5 * n + g * n + 1.75 * (n + n / 2) for n, g in steps)
    assert general["fold_round"] == sum(1.5 * n + 0.75 * (n + n / 2) for n, _ in steps)
    # 2^17: one round over the device, then a launch for the rest
    cfg = lg.ProverConfig(1, (1 << 17, 2), [(1 << 14, 8)], 1, [3])
    poly = lg.splitmix_coeffs_device(2, cfg.poly_len, ctx)
    stats, _, _ = _booked(ctx, lambda: lg.prover(cfg, poly, ctx))
    assert stats["fold_round"][0] == 1 and stats["fold_round_grid"][0] == 1
