"""The last FFT pass on both sides of its rule: tiles by plain loads while there
are fewer than four an SM, by bulk copies from there on; full tiles, ragged ones
and a single vector; 4, 5 and 6 stages, alone and after a strided pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
rng = np.random.default_rng(23)


@pytest.fixture
def split(ctx):
    yield ctx.set_fft_split
    ctx.set_fft_split()


ALONE = [((k,), b) for k in (4, 5, 6) for b in (1, 2, 7, 63, 64, 65, 130, 591 * 64, 591 * 64 + 1, 592 * 64)]
AFTER = [((5, 6), 64 * 18), ((5, 6), 64 * 18 + 1), ((5, 6), 64 * 19), ((4, 4), 64 * 37 + 3), ((3, 5), 5), ((4, 6), 1)]
FEW = [((5, 5, 6), b) for b in (1, 7, 8, 9)]


# 591 and 592 tiles: the last without bulk copies and the first with them; many
# tiles of few vectors, with copies from 8 vectors on
@pytest.mark.parametrize("stages,batch", ALONE + AFTER + FEW)
def test_tiles(lg, ref, ctx, split, stages, batch):
    log_n = sum(stages)
    v = rng.integers(0, 2**32, size=batch << log_n, dtype=np.uint64).astype(np.uint32)
    tw, d = ref.twiddles(log_n), lg.to_device(v)
    split(stages)
    lg.fft(d, log_n, ctx)
    got, src = lg.to_host(d).reshape(batch, -1), v.reshape(batch, -1)
    for i in sorted({0, 1 % batch, batch // 2, max(0, batch - 2), batch - 1}):
        assert (got[i] == ref.fft(src[i], tw=tw)).all()
    lg.ifft(d, log_n, ctx)
    assert (lg.to_host(d) == v).all()


@pytest.mark.parametrize("log_n,batch", [(7, 3), (8, 17), (9, 500), (10, 500), (11, 64), (13, 17), (16, 64), (19, 3)])
@pytest.mark.parametrize("shift", [0, 1])
def test_default_splits(lg, ref, ctx, log_n, batch, shift):
    v = rng.integers(0, 2**32, size=batch << log_n, dtype=np.uint64).astype(np.uint32)
    tw = ref.twiddles(log_n)
    d = lg.to_device(np.concatenate([np.zeros(shift, np.uint32), v]))[shift:]
    lg.fft(d, log_n, ctx)
    got, src = lg.to_host(d).reshape(batch, -1), v.reshape(batch, -1)
    for i in sorted({0, batch // 2, batch - 1}):
        assert (got[i] == ref.fft(src[i], tw=tw)).all()
    lg.ifft(d, log_n, ctx)
    assert (lg.to_host(d) == v).all()
