"""The verifier's openings, checked beside each other in one launch: proofs of
several shapes are accepted, and a byte changed in any opening's rows or
siblings gives the oracle's outcome."""
import pytest

pytestmark = pytest.mark.gpu

# (log_m0, log_n0, [(log_m, log_n)]): trees of 2^8 .. 2^14 leaves, 1 to 3
# openings on the device beside the first, rows of 2 to 256 words
SHAPES = [
    (10, 6, [(6, 4)]), (8, 8, [(7, 1)]), (12, 1, [(9, 3), (6, 3)]), (11, 5, [(10, 1), (8, 2), (6, 2)]),
]


def _spans(p):
    """Byte ranges of every opening's rows and siblings in the encoding."""
    at, out = 12, []

    def u32():
        nonlocal at
        at += 4
        return int.from_bytes(p[at - 4:at], "little")

    def opening():
        nonlocal at
        for _ in range(2):  # rows, then siblings
            spans, words = [], len(out) % 2 == 0
            for _ in range(u32()):
                n = u32() * (4 if words else 1)
                spans.append((at, n))
                at += n
            out.append(spans)

    def skip(unit):
        nonlocal at
        n = u32()
        at += unit * n

    skip(1)
    for _ in range(u32()):
        skip(1)
    opening()
    for _ in range(u32()):
        opening()
    skip(4)
    opening()
    return out


@pytest.mark.parametrize("shape", SHAPES)
def test_openings(lg, ref, ctx, shape):
    lm0, ln0, dims = shape
    pc = lg.ProverConfig(len(dims), (1 << lm0, 1 << ln0), [(1 << m, 1 << n) for m, n in dims], ln0, [n for _, n in dims])
    rc = ref.config(len(dims), lm0, ln0, [m for m, _ in dims], [n for _, n in dims])
    proof = lg.prover(pc, lg.to_device(lg.splitmix_coeffs(77, pc.poly_len)), ctx).to_bytes()
    assert lg.verifier(pc, proof, ctx) and ref.verify(rc, proof) == (0, True)
    for spans in _spans(proof):
        for at, n in {spans[i] for i in (0, len(spans) // 2, len(spans) - 1) if spans}:
            bad = bytearray(proof)
            bad[at + n // 2] ^= 0x10
            want = ref.verify(rc, bytes(bad))
            try:
                got = (0, lg.verifier(pc, bytes(bad), ctx))
            except lg.LigeritoPanic:
                got = (5, False)
            assert got[1] == want[1] and (got[0] == 0) == (want[0] == 0)
