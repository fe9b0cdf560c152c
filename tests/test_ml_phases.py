"""Multilinear proofs from two reads of the table, at the smallest sizes that
run so and around the lines between the integer and the tensor-core sums, both
orders, whole and partial runs, random words and every digit at its largest,
against the oracle.  Exact."""
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


@pytest.mark.parametrize("field", [1, 3])
@pytest.mark.parametrize("order", ["msb", "lsb"])
@pytest.mark.parametrize("n,rounds,top", [(17, 17, False), (18, 18, False), (18, 10, True), (19, 15, False), (20, 20, True),
                                          (21, 21, False), (22, 12, False)])
def test_two_reads(E, n, rounds, top, order, field):
    g = np.random.default_rng(n + field)
    t = np.full(1 << n, 0xFFFFFFFEFFFFFFFF, np.uint64) if top else g.integers(0, O.P, size=1 << n, dtype=np.uint64)
    orc = O.Prover(O.ML, O.LSB if order == "lsb" else O.MSB, field, [t])
    rp, ch, fv = O.sumcheck(orc, rounds, O.Transcript(field, label=b"ml2"), hook=b"\x09\x08")
    pr = (E.MultilinearProverLSB if order == "lsb" else E.MultilinearProver)(t, field=field)
    for use_graph in (True, False):
        pr.reset()
        x = pr.prove(rounds, E.Transcript.keccak(field, b"ml2"), hook=b"\x09\x08", use_graph=use_graph)
        assert np.array_equal(np.asarray(x.round_polys).reshape(rounds, field), rp[:, 0, :field])
        assert np.array_equal(np.asarray(x.challenges).reshape(rounds, field), ch[:, :field])
        assert np.array_equal(np.asarray(x.final_value).reshape(field), fv[:field])
        assert np.array_equal(np.asarray(pr.table(0)).reshape(-1, field), orc.table(0)[:, :field])
