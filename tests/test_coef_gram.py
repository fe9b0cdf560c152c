"""The tensor-core first pass of a degree-3 Coefficient proof (rounds 0-1):
against one pass per round and the oracle where it can go wrong -- the fewest
tiles, every digit at its largest, accumulators filled over several launches,
both orders, table 0 in Fp and Fp3, tables that are not 16-byte aligned.
Everything is exact: no tolerance."""
import os

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOP = 0xFFFFFFFEFFFFFFFF


@pytest.fixture(scope="module")
def E():
    import effsc_gpu
    effsc_gpu.load()
    O.set_threads(os.cpu_count() or 1)
    return effsc_gpu


def tables(n, ext0, what, seed):
    g = np.random.default_rng(seed)
    shape = (1 << n, 3) if ext0 else (1 << n,)
    if what == "top":
        # tables 1 and 2 constant: their products' values are one word with few small digits
        f = np.full(1 << n, 0xEFFFFFFFEFFFFFFF, dtype=np.uint64)
        return [np.full(shape, TOP, dtype=np.uint64), f, np.ones(1 << n, dtype=np.uint64)]
    return [g.integers(0, O.P, size=shape, dtype=np.uint64)] + [g.integers(0, O.P, size=1 << n, dtype=np.uint64) for _ in range(2)]


def check(pf, tabs, order, rounds):
    rp, ch, fv = O.sumcheck(O.Prover(O.COEF, order, 3, tabs), rounds, O.Transcript(3, label=b"c3g"), hook=b"\x09" * 8)
    assert np.array_equal(pf.round_polys, rp) and np.array_equal(pf.challenges, ch) and np.array_equal(pf.final_value, fv)


@pytest.mark.parametrize("lsb", [False, True])
@pytest.mark.parametrize("ext0", [False, True])
@pytest.mark.parametrize("n,what", [(12, "uniform"), (13, "top"), (17, "uniform"), (19, "top")])
def test_proofs(E, lsb, ext0, n, what):
    tabs = tables(n, ext0, what, n + ext0)
    p = (E.CoefficientProverLSB if lsb else E.CoefficientProver)(tabs)
    check(p.prove(5, E.Transcript.keccak(E.FP3, b"c3g"), hook=b"\x09" * 8), tabs, O.LSB if lsb else O.MSB, 5)


@pytest.mark.parametrize("what", ["top", "uniform"])
def test_full_accumulators(E, what):
    tabs = tables(26, False, what, 3)
    check(E.CoefficientProver(tabs).prove(3, E.Transcript.keccak(E.FP3, b"c3g"), hook=b"\x09" * 8), tabs, O.MSB, 3)


@pytest.mark.parametrize("lsb", [False, True])
def test_unaligned(E, lsb):
    import torch
    n = 14
    tabs = tables(n, False, "uniform", 8)
    dev = []
    for t in tabs:
        d = torch.empty((1 << n) + 1, dtype=torch.int64, device="cuda")
        d[1:] = torch.from_numpy(t.view(np.int64)).cuda()
        dev.append(d)
    torch.cuda.synchronize()
    cls = E.CoefficientProverLSB if lsb else E.CoefficientProver
    p = cls.from_device([d.data_ptr() + 8 for d in dev], [1 << n] * 3, [1, 1, 1])
    check(p.prove(5, E.Transcript.keccak(E.FP3, b"c3g"), hook=b"\x09" * 8), tabs, O.LSB if lsb else O.MSB, 5)
