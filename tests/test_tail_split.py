"""The tail kernels' splits: a cluster from the first round on (groups of 4
and of 16 entries, MSB and LSB), a hand-over at the last round of a partial
run, the one-product, row and whole-value roles of the round polynomial, and
transcript hooks that do and do not fit one block -- against the oracle,
proofs and post-state tables."""
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


CASES = [(k, o, f, n, n) for k in ("ip", "ml") for o in ("msb", "lsb") for f in (1, 3) for n in (1, 5, 6, 7, 10, 11, 12, 13, 16)]
CASES += [("ip", o, 3, n, r) for o in ("msb", "lsb") for n, r in ((11, 4), (11, 5), (11, 6), (12, 6), (14, 6), (14, 7), (17, 9))]


@pytest.mark.parametrize("kind,order,field,n,rounds", CASES)
def test_split(E, kind, order, field, n, rounds):
    k = 2 if kind == "ip" else 1
    g = np.random.default_rng(1000 * n + 10 * rounds + field)
    tabs = [g.integers(0, O.P, size=1 << n, dtype=np.uint64) for _ in range(k)]
    cls = {("ip", "msb"): E.InnerProductProver, ("ip", "lsb"): E.InnerProductProverLSB,
           ("ml", "msb"): E.MultilinearProver, ("ml", "lsb"): E.MultilinearProverLSB}[kind, order]
    for hook in (b"", bytes(range(88)), bytes(range(96)), b"\x05" * 13):
        p = cls(*tabs, field=field)
        pf = p.prove(rounds, E.Transcript.keccak(field, b"split"), hook=hook)
        orc = O.Prover(O.IP if kind == "ip" else O.ML, O.MSB if order == "msb" else O.LSB, field, tabs)
        rp, ch, fv = O.sumcheck(orc, rounds, O.Transcript(field, label=b"split"), hook=hook)
        assert np.array_equal(np.asarray(pf.round_polys).reshape(rounds, k, field), rp[:, :k, :field])
        assert np.array_equal(np.asarray(pf.challenges).reshape(rounds, field), ch[:, :field])
        assert np.array_equal(np.asarray(pf.final_value).reshape(field), fv[:field])
        for t in range(k):
            assert np.array_equal(np.asarray(p.table(t)).reshape(-1, field), orc.table(t)[:, :field])
