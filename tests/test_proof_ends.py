"""Hooks around the length that travels with the transcript's state (512
bytes), of whole words and not, in one prover after another length, against
the oracle.  Exact."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", [1, 3])
@pytest.mark.parametrize("use_graph", [True, False])
def test_hook_lengths(field, use_graph):
    import effsc_gpu as E
    E.load()
    g = np.random.default_rng(field)
    a, b = (g.integers(0, O.P, size=1 << 9, dtype=np.uint64) for _ in range(2))
    pr = E.InnerProductProver(a, b, field=field)
    for n in (0, 1, 511, 512, 513, 7, 520, 1200, 8):
        hook = bytes((3 * i + n) % 256 for i in range(n))
        pr.reset()
        x = pr.prove(9, E.Transcript.keccak(field, b"ends"), hook=hook, use_graph=use_graph)
        rp, ch, fv = O.sumcheck(O.Prover(O.IP, O.MSB, field, [a, b]), 9, O.Transcript(field, label=b"ends"), hook=hook)
        assert np.array_equal(np.asarray(x.round_polys).reshape(9, 2, field), rp[:, :2, :field]), n
        assert np.array_equal(np.asarray(x.challenges).reshape(9, field), ch[:, :field]), n
        assert np.array_equal(np.asarray(x.final_value).reshape(field), fv[:field]), n
