"""Sumcheck steps that run in one launch (a cluster per proof), against the
oracle's proofs: step sizes from the smallest to past the largest that fits,
one to six rounds a step, clusters of one to eight blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (log of the folded vector, rounds of each step): the first step's words
# 2^7 .. 2^17 cover one block, partly filled clusters, the largest step in one
# launch (2^16) and one whose first round runs alone (2^17); later steps glue
CASES = [
    (7, [1]), (8, [2]), (10, [4]), (11, [1, 1, 2]), (12, [6]), (13, [2, 4]), (14, [3, 4]), (15, [1, 4]),
    (16, [5, 4]), (17, [2, 1, 4]),
]


def _configs(lg, ref, log_m, ks):
    dims, left = [], log_m
    for k in ks:
        left -= k
        dims.append((left, k))
    pc = lg.ProverConfig(len(ks), (1 << log_m, 2), [(1 << m, 1 << n) for m, n in dims], 1, list(ks))
    rc = ref.config(len(ks), log_m, 1, [m for m, _ in dims], list(ks))
    return pc, rc


@pytest.mark.parametrize("log_m,ks", CASES)
def test_steps_match_oracle(lg, ref, ctx, log_m, ks):
    pc, rc = _configs(lg, ref, log_m, ks)
    poly = lg.splitmix_coeffs(31 + log_m, pc.poly_len)
    assert lg.prover(pc, lg.to_device(poly), ctx).to_bytes() == ref.prove(rc, poly, nthreads=8)


@pytest.mark.parametrize("log_m,ks,B", [(10, [4], 64), (14, [3, 4], 9), (14, [3, 4], 19), (16, [5, 4], 3)])
def test_lockstep_steps_match_single(lg, ref, ctx, log_m, ks, B):
    # the batch sets the clusters' size (as many blocks as the device holds)
    pc, rc = _configs(lg, ref, log_m, ks)
    polys = np.stack([lg.splitmix_coeffs(900 + b, pc.poly_len) for b in range(B)])
    got = lg.prove_lockstep(pc, lg.to_device(polys.ravel()).view(B, -1), ctx)
    for b in (0, B // 2, B - 1):
        assert got[b].to_bytes() == ref.prove(rc, polys[b], nthreads=8)


@pytest.mark.parametrize("k0", [2, 3, 4, 5, 7, 8])
def test_first_challenges_match_oracle(lg, ref, ctx, k0):
    # the number of challenges squeezed at once moves every later word of the
    # transcript inside its SHA-256 blocks
    pc = lg.ProverConfig(2, (1 << 10, 1 << k0), [(1 << 8, 4), (1 << 6, 4)], k0, [2, 2])
    rc = ref.config(2, 10, k0, [8, 6], [2, 2])
    poly = lg.splitmix_coeffs(50 + k0, pc.poly_len)
    assert lg.prover(pc, lg.to_device(poly), ctx).to_bytes() == ref.prove(rc, poly, nthreads=8)
