"""Pinned polynomials of the largest size that travels whole (2^20 words) and
the first in groups (2^21), with few and many columns, give the device input's
proof."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log", [20, 21])
@pytest.mark.parametrize("cols", [1, 4, 5, 7, 8])
def test_pinned_input(lg, ctx, log, cols):
    dims, left = [], log - cols
    while not dims or left - 4 >= 10:
        left -= 4
        dims.append((1 << left, 16))
    cfg = lg.ProverConfig(len(dims), (1 << (log - cols), 1 << cols), dims, cols, [4] * len(dims))
    dev = lg.splitmix_coeffs_device(log, 1 << log, ctx)
    host = dev.cpu().pin_memory().numpy().view(np.uint32)
    assert lg.prover(cfg, host, ctx).to_bytes() == lg.prover(cfg, dev, ctx).to_bytes()
