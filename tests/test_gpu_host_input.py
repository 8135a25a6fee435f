"""Host polynomials: the whole copy of small ones and the grouped copy of the
others, on both sides of each limit, give the proof of the device input."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [16, 18, 19, 21, 22])
def test_host_inputs_give_the_device_inputs_proof(lg, ctx, L):
    import torch

    cfg = lg.config_for_size(L)
    dev = lg.splitmix_coeffs_device(L, 1 << L, ctx)
    want = lg.prover(cfg, dev, ctx).to_bytes()
    pageable = dev.cpu()
    for host in (pageable, pageable.pin_memory()):
        assert lg.prover(cfg, host.numpy().view(np.uint32), ctx).to_bytes() == want
