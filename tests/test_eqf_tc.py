"""EqFactoredProver's left phase over base tables large enough for the
tensor-core sums (one and several blocks per group of entries, odd and even
v, Fp and Fp3, weights all in Fp, every digit at its largest) against the
oracle: proofs and the tables after full and partial runs.  Exact."""
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


@pytest.mark.parametrize("field,wext", [(3, True), (3, False), (1, False)])
@pytest.mark.parametrize("v,rounds,top", [(17, 17, False), (18, 9, False), (18, 18, True), (19, 19, False), (20, 12, False),
                                          (21, 21, False), (22, 11, True)])
def test_left_phase(E, field, wext, v, rounds, top):
    g = np.random.default_rng(10 * v + field)
    w = g.integers(0, O.P, size=(v, field), dtype=np.uint64)
    if not wext and field == 3:
        w[:, 1:] = 0
    p = np.full(1 << v, 0xFFFFFFFEFFFFFFFF, dtype=np.uint64) if top else g.integers(0, O.P, size=1 << v, dtype=np.uint64)
    w = w if field == 3 else w.reshape(-1)
    pr = E.EqFactoredProver(w, p, field=field)
    pf = pr.prove(rounds, E.Transcript.keccak(field, b"eqftc"), hook=b"\x01\x02")
    orc = O.Prover.eq_factored(field, w, p)
    rp, ch, fv = O.sumcheck(orc, rounds, O.Transcript(field, label=b"eqftc"), hook=b"\x01\x02")
    assert np.array_equal(np.asarray(pf.round_polys).reshape(rounds, 2, field), rp[:, :2, :field])
    assert np.array_equal(np.asarray(pf.challenges).reshape(rounds, field), ch[:, :field])
    assert np.array_equal(np.asarray(pf.final_value).reshape(field), fv[:field])
    for t in range(3):
        assert np.array_equal(np.asarray(pr.table(t)).reshape(-1, field), orc.table(t)[:, :field]), t
