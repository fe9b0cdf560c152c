"""An admission that fails part of the way: the requests admitted before it are
active, and their proofs are the oracle's once there is room for the one
that failed."""
import os

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_requests_before_a_failed_one():
    import torch
    import effsc_gpu as E
    O.set_threads(os.cpu_count() or 1)
    n, big = 22, 32                  # the same lane; the second of 2^32 x 20 bytes (Multilinear over Fp3)
    need = (1 << big) * 20
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    if free < need + (8 << 30):
        pytest.skip("%d GB free" % (free >> 30))
    srv = E.Server(1 << 38, max_active=8)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (need >> 1), dtype=torch.uint8, device="cuda")
    seeds = [E.table_seed(7, 0), E.table_seed(7, 1)]
    first = srv.submit(E.IP, n, E.Transcript.keccak(E.FP3, b"first"), seeds=seeds)
    srv.submit(E.ML, big, E.Transcript.keccak(E.FP3, b"big"), seeds=[E.table_seed(8, 0)])
    with pytest.raises(E.EffscError) as e:
        srv.progress()
    assert e.value.status == 2       # out of device memory
    del hold
    torch.cuda.empty_cache()
    got = srv.drain()
    pf = got[first][0]
    tabs = [E.gen_uniform(s, 1 << n) for s in seeds]
    rp, ch, fv = O.sumcheck(O.Prover(O.IP, O.MSB, 3, tabs), n, O.Transcript(3, label=b"first"))
    assert len(got) == 2
    assert np.array_equal(pf.round_polys, rp) and np.array_equal(pf.challenges, ch) and np.array_equal(pf.final_value, fv)
    del srv
