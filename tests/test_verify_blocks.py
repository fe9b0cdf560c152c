"""The batch verifier where its loops and buffers change form: proofs of 31 to
65 rounds (the claim is updated 32 rounds at a time), words at and above the
modulus, and a batch above the size that is read in place, against the host's
verifier.  Exact."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import effsc_gpu
    effsc_gpu.load()
    return effsc_gpu


@pytest.mark.parametrize("field", [1, 3])
@pytest.mark.parametrize("degree", [0, 1, 2, 3])
@pytest.mark.parametrize("rounds", [[31, 32, 33, 64, 65, 0, 1], [6] * 30000])
def test_blocks(E, field, degree, rounds):
    g = np.random.default_rng(degree + 10 * field + len(rounds))
    n, nw = len(rounds), max(degree, 1)
    claims = g.integers(0, O.P, size=(n, field), dtype=np.uint64)
    polys = [g.integers(0, O.P, size=(r, nw, field), dtype=np.uint64) for r in rounds]
    for p in polys[:5]:
        p[0] = 0xFFFFFFFFFFFFFFFF      # 2^32 - 2 as a residue
        p[1:3] = O.P
    claims[0] = 0xFFFFFFFF00000001
    labels = [b"vbl/%d" % i for i in range(n)]
    fin, chs = E.sumcheck_verify_batch(claims, degree, polys, [E.Transcript.keccak(field, x) for x in labels],
                                       hook=b"\x07" * 8, field=field)
    assert len(chs) == n
    for i in range(n) if n < 100 else range(0, n, 1499):
        ch, fc = E.sumcheck_verify(list(claims[i] % np.uint64(O.P)), degree, rounds[i], E.Transcript.keccak(field, labels[i]),
                                   polys[i] % np.uint64(O.P), hook=b"\x07" * 8)
        assert np.array_equal(chs[i], ch.reshape(-1, field)), i
        assert np.array_equal(fin[i], fc), i
