"""Tables from pageable host memory (a served request's are copied by a kernel
from 64 KB on): lengths around that limit, odd lengths, sources 8 but not 16
bytes aligned, memory the caller changes as soon as the call returns, and
served requests from such tables of every size around the tensor-core start's
and the tail's limits -- against the oracle."""
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


@pytest.mark.parametrize("n", [8191, 8192, 8193, 20001, 1 << 15])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("ncomp", [1, 3])
def test_tables(E, n, shift, ncomp):
    g = np.random.default_rng(n + shift)
    shape = (n,) if ncomp == 1 else (n, 3)
    raw = np.empty(n * ncomp + 2, dtype=np.uint64)
    off = ((raw.ctypes.data // 8) + shift) % 2
    t = raw[off:off + n * ncomp].reshape(shape)
    t[...] = g.integers(0, O.P, size=shape, dtype=np.uint64)
    keep = t.copy()
    p = E.MultilinearProver(t)
    t[...] = 0                      # the prover has its copy
    got = p.evals()
    assert np.array_equal(got[:, 0] if ncomp == 1 else got, keep)


def test_serving(E):
    g = np.random.default_rng(3)
    srv = E.Server(8 << 30, max_active=16)
    want = {}
    for i, n in enumerate([1, 5, 12, 13, 14, 15, 16, 17, 18, 19, 14, 20]):
        tabs = [g.integers(0, O.P, size=1 << n, dtype=np.uint64) for _ in range(2)]
        label = b"up%d" % i
        rid = srv.submit(E.IP, n, E.Transcript.keccak(E.FP3, label), tables=tabs)
        want[rid] = O.sumcheck(O.Prover(O.IP, O.MSB, 3, tabs), n, O.Transcript(3, label=label))
    got = srv.drain()
    for rid, (rp, ch, fv) in want.items():
        pf = got[rid][0]
        assert np.array_equal(pf.round_polys, rp) and np.array_equal(pf.challenges, ch) and np.array_equal(pf.final_value, fv)
