"""The degree-3 Coefficient tail (one block, a cluster, and the sizes between
which the kernels change) against the per-round path and the oracle: proofs,
the tables after whole and partial runs, both orders, base and Fp3 first
tables, hooks.  Exact."""
import os

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import effsc_gpu
    effsc_gpu.load()
    O.set_threads(os.cpu_count() or 1)
    return effsc_gpu


@pytest.mark.parametrize("lsb", [False, True])
@pytest.mark.parametrize("ext", [0, 1, 3])
@pytest.mark.parametrize("n,rounds", [(2, 2), (3, 2), (6, 6), (9, 4), (11, 11), (12, 12), (12, 5), (13, 8), (15, 15), (16, 10)])
def test_tail(E, lsb, ext, n, rounds):
    g = np.random.default_rng(100 * n + rounds + ext)
    tabs = [g.integers(0, O.P, size=(1 << n, 3) if i < ext else 1 << n, dtype=np.uint64) for i in range(3)]
    hook = bytes(range(n))
    orc = O.Prover(O.COEF, O.LSB if lsb else O.MSB, 3, tabs)
    rp, ch, fv = O.sumcheck(orc, rounds, O.Transcript(3, label=b"c3t"), hook=hook)
    for tail in (None, 64, 0):
        p = (E.CoefficientProverLSB if lsb else E.CoefficientProver)(tabs)
        p.set_tail(tail)
        pf = p.prove(rounds, E.Transcript.keccak(E.FP3, b"c3t"), hook=hook)
        assert np.array_equal(pf.round_polys, rp), tail
        assert np.array_equal(pf.challenges, ch) and np.array_equal(pf.final_value, fv), tail
        for t in range(3):
            assert np.array_equal(np.asarray(p.table(t)).reshape(-1, 3), orc.table(t)), (tail, t)
