"""Whole GkrProver proofs from two reads of the gate tables: at the smallest
size that runs so, on both sides of the line between the integer and the
tensor-core sums, with random words and with every digit at its largest (the
witness zero or the largest residue), against the oracle and the per-round
path, the four tables after the run included.  Exact."""
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
@pytest.mark.parametrize("k,words", [(4, "random"), (5, "top"), (9, "zero"), (10, "random"), (10, "top"), (11, "random"),
                                     (11, "top"), (11, "zero")])
def test_two_reads(E, k, words, field):
    n, top = 1 << k, 0xFFFFFFFEFFFFFFFF      # a residue whose digits are 14 and 15
    g = np.random.default_rng(40 * k + field)
    draw = lambda m: g.integers(0, O.P, size=m, dtype=np.uint64)  # noqa: E731
    add, mult = (np.full(n * n, top, np.uint64) if words == "top" else draw(n * n) for _ in range(2))
    w = np.full(n, top, np.uint64) if words == "top" else np.zeros(n, np.uint64) if words == "zero" else draw(n)
    hook = b"\x01\x02\x03" if k % 2 else b""
    rp, ch, fv = O.sumcheck(O.Prover.gkr(field, add, mult, w), 2 * k, O.Transcript(field, label=b"2r"), hook=hook)
    tables = []
    for first, use_graph in ((True, True), (True, False), (False, False)):
        p = E.GkrProver(add, mult, w, field=field)
        p.set_first_rounds(first)
        for _ in range(2):
            p.reset()
            x = p.prove(2 * k, E.Transcript.keccak(field, b"2r"), hook=hook, use_graph=use_graph)
            assert np.array_equal(np.asarray(x.round_polys).reshape(2 * k, 2, field), rp[:, :2, :field])
            assert np.array_equal(np.asarray(x.challenges).reshape(2 * k, field), ch[:, :field])
            assert np.array_equal(np.asarray(x.final_value).reshape(field), fv[:field])
        tables.append([np.asarray(p.table(t)) for t in range(4)] + [p.claimed_w_values()])
    for other in tables[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(tables[0], other))
