"""Digit sums to the last bit: the tensor-core passes add products of 4-bit
digits in f32, exact while the sums stay below 2^24.  Constant tables make all
of a 32-term instruction's products alike, and uniform ones stay far below
that; here every digit is 14 or 15 at random (the top one 14: residues), so that
the sums of a block's accumulator are odd as often as even, up to
65536 x 225.  Four rounds of 2^27 entries fill the accumulators (512 tiles a
block of 152 in the first of two launches), five take 432 tiles: a bit lost
anywhere below 2^24 would show.  Against the oracle; exact."""
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


def high(g, *shape):
    """Words of digits 14 and 15, the top one 14 (below p)."""
    w = g.integers(0, 1 << 64, size=shape, dtype=np.uint64)
    w &= np.uint64(0x0111111111111111)
    w |= np.uint64(0xEEEEEEEEEEEEEEEE)
    return w


@pytest.mark.parametrize("n,order,rounds", [(26, "msb", 5), (27, "msb", 4), (27, "msb", 5), (27, "lsb", 5)])
def test_inner_product(E, n, order, rounds):
    g = np.random.default_rng(n + rounds)
    tabs = [high(g, 1 << n) for _ in range(2)]
    cls = E.InnerProductProver if order == "msb" else E.InnerProductProverLSB
    pf = cls(*tabs).prove(rounds, E.Transcript.keccak(E.FP3, b"digits"))
    rp, ch, fv = O.sumcheck(O.Prover(O.IP, O.MSB if order == "msb" else O.LSB, 3, tabs), rounds, O.Transcript(3, label=b"digits"))
    assert np.array_equal(pf.round_polys, rp) and np.array_equal(pf.challenges, ch) and np.array_equal(pf.final_value, fv)


@pytest.mark.parametrize("n,ext0,order", [(25, False, "msb"), (25, True, "msb"), (25, False, "lsb")])
def test_coefficient(E, n, ext0, order):
    """Table 2 is all ones: the products' values at the four corners of a quadruple
    are table 1's words, digits of 14 and 15 as table 0's."""
    g = np.random.default_rng(n + ext0)
    tabs = [high(g, 1 << n, 3) if ext0 else high(g, 1 << n), high(g, 1 << n), np.ones(1 << n, dtype=np.uint64)]
    cls = E.CoefficientProver if order == "msb" else E.CoefficientProverLSB
    pf = cls(tabs).prove(3, E.Transcript.keccak(E.FP3, b"digits"))
    rp, ch, fv = O.sumcheck(O.Prover(O.COEF, O.MSB if order == "msb" else O.LSB, 3, tabs), 3, O.Transcript(3, label=b"digits"))
    assert np.array_equal(pf.round_polys, rp) and np.array_equal(pf.challenges, ch) and np.array_equal(pf.final_value, fv)
