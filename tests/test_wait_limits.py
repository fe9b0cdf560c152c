"""The tensor-core passes' waits run out, without a fault.

Their pipelines (k_ip_gram, k_tc_fold, k_c3_gram, k_eqf_tc) wait between their
warps with a limit.  Here the limit is zero for the loading and the epilogue
warps, so that they give up where a stage is not free, or its sums are not there,
yet (the sizes give every block more tiles than stages): the pass has to end by
itself, its tensor memory given back and its warps together, the call has to
say EFFSC_TIMEOUT, and the same prover's next proof, with the usual limit, has
to be the oracle's, word for word."""
import os

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
LABEL = b"limits"


@pytest.fixture(scope="module")
def E():
    import effsc_gpu
    effsc_gpu.load()
    O.set_threads(os.cpu_count() or 1)
    return effsc_gpu


def cases(E, what):
    """(prover, rounds, oracle prover)"""
    g = np.random.default_rng(len(what))

    def words(*shape):
        return g.integers(0, O.P, size=shape, dtype=np.uint64)
    if what.startswith("ip"):
        lsb, rounds = "lsb" in what, 4 if "four" in what else 21
        tabs = [words(1 << 21) for _ in range(2)]
        return (E.InnerProductProverLSB if lsb else E.InnerProductProver)(*tabs), rounds, O.Prover(O.IP, O.LSB if lsb else O.MSB, 3, tabs)
    if what.startswith("ml"):
        lsb, n = "lsb" in what, 21
        t = words(1 << n)
        return (E.MultilinearProverLSB if lsb else E.MultilinearProver)(t), n, O.Prover(O.ML, O.LSB if lsb else O.MSB, 3, [t])
    if what.startswith("coef"):
        lsb = "lsb" in what
        tabs = [words(1 << 20, 3), words(1 << 20), words(1 << 20)]
        return (E.CoefficientProverLSB if lsb else E.CoefficientProver)(tabs), 20, O.Prover(O.COEF, O.LSB if lsb else O.MSB, 3, tabs)
    if what == "eqf":
        w, p = words(21, 3), words(1 << 21)
        return E.EqFactoredProver(w, p), 21, O.Prover.eq_factored(3, w, p)
    n = 1 << 11
    add, mult, w = words(n * n), words(n * n), words(n)
    return E.GkrProver(add, mult, w), 22, O.Prover.gkr(3, add, mult, w)


@pytest.mark.parametrize("what", ["ip", "ip lsb", "ip four", "ml", "ml lsb", "coef", "coef lsb", "eqf", "gkr"])
def test_gives_up_and_proves_again(E, what):
    p, rounds, orc = cases(E, what)
    rp, ch, fv = O.sumcheck(orc, rounds, O.Transcript(3, label=LABEL))

    def no_wait(on):
        E.api.check(E.load().effsc_diag_prover_no_wait(p.h, on))
    for graph in (False, True):
        no_wait(1)
        for _ in range(2):
            t = E.Transcript.keccak(3, LABEL)
            with pytest.raises(E.EffscError) as e:
                p.prove(rounds, t, use_graph=graph)
            assert e.value.status == 4
            assert t.squeeze(16) == E.Transcript.keccak(3, LABEL).squeeze(16)      # as it was
            p.reset()
        no_wait(0)
        for _ in range(2):
            pf = p.prove(rounds, E.Transcript.keccak(3, LABEL), use_graph=graph)
            assert np.array_equal(pf.round_polys, rp[:, :pf.round_polys.shape[1]])
            assert np.array_equal(pf.challenges, ch) and np.array_equal(pf.final_value, fv)
            p.reset()
