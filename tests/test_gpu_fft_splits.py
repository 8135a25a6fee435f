"""Every kind of FFT pass that a stage split can hold, whoever chooses it (the
autotuner may take strided passes of 5 and 6 stages, and an encoding's first
pass of 5), bit for bit against the oracle: rows by bulk copies and not, data
that is only word-aligned, ragged vector counts, few units and many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
rng = np.random.default_rng(17)


def rand_u32(n):
    return rng.integers(0, 2**32, size=n, dtype=np.uint64).astype(np.uint32)


def on_device(lg, v, shift):
    """v on the device, `shift` words past an aligned address."""
    return lg.to_device(np.concatenate([np.zeros(shift, np.uint32), v]))[shift:]


@pytest.fixture
def split(ctx):
    yield ctx.set_fft_split
    ctx.set_fft_split()


def passes_run(ctx, call):
    """stages of the passes that a call ran, largest first"""
    ctx.set_kernel_timing(True)
    ctx.reset_kernel_stats()
    try:
        call()
        return sorted(sum(([int(k.split("_K")[1].split("_")[0])] * n for k, (n, _) in ctx.kernel_stats().items()
                           if "_K" in k), []), reverse=True)
    finally:
        ctx.set_kernel_timing(False)
        ctx.reset_kernel_stats()


# first and later passes of 5 and 6, rows of 2^S >= 32 words (bulk copies) and
# fewer, rows longer than a block, last passes of 1..3 stages (strided too)
SPLITS = [(5, 5), (6, 5), (5, 6), (6, 6), (6, 4), (3, 5, 4), (2, 6, 4), (5, 5, 5), (6, 6, 4), (4, 6, 6), (5, 3), (6, 2), (6, 6, 1)]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("batch", [1, 37])
@pytest.mark.parametrize("stages", SPLITS)
def test_transform(lg, ref, ctx, split, stages, batch, shift):
    log_n = sum(stages)
    v, tw = rand_u32(batch << log_n), ref.twiddles(log_n)
    d = on_device(lg, v, shift)
    split(stages)
    assert passes_run(ctx, lambda: lg.fft(d, log_n, ctx)) == sorted(stages, reverse=True)
    got, src = lg.to_host(d).reshape(batch, -1), v.reshape(batch, -1)
    for i in sorted({0, batch // 2, batch - 1}):
        assert (got[i] == ref.fft(src[i], tw=tw)).all()
    lg.ifft(d, log_n, ctx)
    assert (lg.to_host(d) == v).all()


# many more units than the device holds at once
@pytest.mark.parametrize("stages,batch", [((5, 6), 1201), ((6, 5), 1201), ((5, 5, 6), 130)])
def test_many_units(lg, ref, ctx, split, stages, batch):
    test_transform(lg, ref, ctx, split, stages, batch, 0)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [1, 40])
@pytest.mark.parametrize("stages", [(5, 4), (5, 6), (5, 5, 4), (1, 6), (2, 5, 5), (3, 6, 6), (4, 6, 5), (5, 2)])
def test_encode(lg, ref, ctx, split, stages, n, shift):
    log_m = sum(stages)
    poly = rand_u32(n << log_m)
    src = on_device(lg, poly, shift)
    split(stages)
    out = []
    assert passes_run(ctx, lambda: out.append(lg.encode_cols(src, log_m, n, ctx))) == sorted(stages, reverse=True)
    enc = lg.to_host(out[0]).reshape(n, -1)
    for j in sorted({0, n // 2, n - 1}):
        v = np.zeros(4 << log_m, np.uint32)
        v[: 1 << log_m] = poly[j << log_m : (j + 1) << log_m]
        assert ref.lib().lgref_rs_encode_non_systematic(32, v.ctypes.data, 1 << log_m, 4 << log_m, 4) == 0
        assert (enc[j] == v).all()


def test_what_is_refused(lg, ctx, split):
    for bad in [(0, 5), (7,), (1,) * 7]:
        with pytest.raises(lg.LigeritoError) as e:
            split(bad)
        assert e.value.status == 1
    split((6, 4))
    poly = lg.splitmix_coeffs_device(1, 3 << 10, ctx)
    with pytest.raises(lg.LigeritoError) as e:
        lg.encode_cols(poly, 10, 3, ctx)  # a first pass of 6 stages
    assert e.value.status == 4
    split()
    lg.encode_cols(poly, 10, 3, ctx)
