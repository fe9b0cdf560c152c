"""The tensor-core first pass of an InnerProduct proof (rounds 0-2 from a Gram
matrix of 4-bit digits): whole proofs against the oracle where it can go
wrong -- the fewest tiles, every digit at its largest over the most octets an
accumulator takes, more octets than that (several launches), tables with
zeros and single words, LSB order, host tables (copied on the way, and
uploaded in chunks), and tables that are not 16-byte aligned (the general
pass).  Everything is exact: no tolerance."""
import os

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOP = 0xFFFFFFFEFFFFFFFF      # all digits 15 but one: the largest sums


@pytest.fixture(scope="module")
def E():
    import effsc_gpu
    effsc_gpu.load()
    O.set_threads(os.cpu_count() or 1)
    return effsc_gpu


def tables(n, what, seed):
    g = np.random.default_rng(seed)
    if what == "uniform":
        return [g.integers(0, O.P, size=1 << n, dtype=np.uint64) for _ in range(2)]
    if what == "top":
        return [np.full(1 << n, TOP, dtype=np.uint64), np.full(1 << n, O.P - 1, dtype=np.uint64)]
    if what == "top2":
        return [np.full(1 << n, TOP, dtype=np.uint64) for _ in range(2)]
    a, b = np.zeros(1 << n, dtype=np.uint64), np.zeros(1 << n, dtype=np.uint64)
    for j in range(64):          # one word each, spread over the table
        a[(j * 7919 * 64 + j) % (1 << n)] = g.integers(1, O.P, dtype=np.uint64)
        b[(j * 7919 * 64 + j) % (1 << n)] = g.integers(1, O.P, dtype=np.uint64)
    return [a, b]


def oracle_proof(tabs, order, rounds):
    return O.sumcheck(O.Prover(O.IP, order, 3, tabs), rounds, O.Transcript(3, label=b"gram"))


def same(pf, want):
    rp, ch, fv = want
    return (np.array_equal(pf.round_polys, rp) and np.array_equal(pf.challenges, ch)
            and np.array_equal(pf.final_value, fv))


@pytest.mark.parametrize("lsb", [False, True])
@pytest.mark.parametrize("n,what", [(17, "uniform"), (18, "top2"), (18, "sparse"), (19, "uniform"), (20, "top"), (21, "sparse")])
def test_proofs(E, lsb, n, what):
    tabs = tables(n, what, n)
    cls = E.InnerProductProverLSB if lsb else E.InnerProductProver
    want = oracle_proof(tabs, O.LSB if lsb else O.MSB, n)
    assert same(cls(*tabs).prove(n, E.Transcript.keccak(E.FP3, b"gram")), want)
    p = cls.from_host(tabs)
    for _ in range(2):           # from the host, then from the copy the first pass made
        assert same(p.prove(n, E.Transcript.keccak(E.FP3, b"gram"), use_graph=False), want)
        p.reset()


@pytest.mark.parametrize("n,what", [(26, "top2"), (27, "top2"), (27, "uniform")])
def test_full_accumulators(E, n, what):
    tabs = tables(n, what, n)
    p = E.InnerProductProver(*tabs)
    assert same(p.prove(4, E.Transcript.keccak(E.FP3, b"gram")), oracle_proof(tabs, O.MSB, 4))


@pytest.mark.parametrize("lsb", [False, True])
def test_unaligned_and_pinned(E, lsb):
    import torch
    n = 18
    tabs = tables(n, "uniform", 5)
    cls = E.InnerProductProverLSB if lsb else E.InnerProductProver
    want = oracle_proof(tabs, O.LSB if lsb else O.MSB, n)
    dev = []
    for t in tabs:
        d = torch.empty((1 << n) + 1, dtype=torch.int64, device="cuda")
        d[1:] = torch.from_numpy(t.view(np.int64)).cuda()
        dev.append(d)
    torch.cuda.synchronize()
    p = cls.from_device([d.data_ptr() + 8 for d in dev], [1 << n] * 2, [1, 1])
    assert same(p.prove(n, E.Transcript.keccak(E.FP3, b"gram")), want)
    pinned = [torch.from_numpy(t.view(np.int64)).pin_memory() for t in tabs]
    p = cls.from_host([t.numpy().view(np.uint64) for t in pinned])
    assert same(p.prove(n, E.Transcript.keccak(E.FP3, b"gram"), use_graph=False), want)


@pytest.mark.parametrize("tail", [None, 0, 64])
def test_batch_start(E, tail):
    """A cohort whose larger instances share the two tensor-core launches
    (one and several blocks each; tables behind odd-sized neighbours)."""
    nv = [1, 14, 16, 3, 17, 15, 2, 19, 13, 18, 16]
    tabs = [tables(v, "uniform", 50 + i) for i, v in enumerate(nv)]
    b = E.Batch(E.IP, nv, tables=tabs)
    b.set_tail(tail)
    for rep in range(2):
        proofs = b.prove([E.Transcript.keccak(E.FP3, b"gram") for _ in nv], use_graph=rep == 1)
        for pf, t, v in zip(proofs, tabs, nv):
            assert same(pf, oracle_proof(t, O.MSB, v)), v
