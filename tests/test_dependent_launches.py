"""Kernels that a dependent launch may start while the kernel before them still
runs: none of them may promise that its input is read-only, and proofs and folds are
the same words under every launch form (EFFSC_PDL unset: the kernels of a few
blocks; 0: none; 1: the whole chain)."""
import glob
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "efficient-sumcheck_gb300", "csrc")


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            yield os.path.basename(path), re.sub(r"//[^\n]*", "", f.read())


def test_dependent_kernels_read_coherently():
    found = 0
    for name, text in sources():
        for m in re.finditer(r"__global__[^;{]*\{", text):
            body = text[m.end():]
            body = body[:body.index("\n}")]
            if "chain_enter();" in body:
                found += 1
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", m.group(0)), (name, m.group(0))
        # bodies shared by several kernels: the InnerProduct start's octets alone
        # are loaded as read-only data
        assert "__ldg(" not in text, name
        assert text.count("ld.global.nc") == (1 if name == "ip012.cuh" else 0), name
    assert found >= 30


def test_a_copied_table_is_read_after_a_plain_launch():
    text = dict(sources())
    for name, fn in (("k_ip012.cu", "launch_ip3x"), ("k_tcfold.cu", "fold_inst")):
        body = text[name][text[name].index("bool %s(" % fn):]
        body = body[:body.index("\n}")]
        assert "pdl_on(false) && !copied" in body and "launch_chain" not in body, name
    calls = re.findall(r"launch_(?:ip3x|tc_fold)\(([^;]*);", text["runtime.cu"])
    assert len(calls) == 2 and all("mirror" in c for c in calls)


CHILD = r"""
import hashlib, sys
import numpy as np
import effsc_gpu as E
g = np.random.default_rng(5)
P = 2**64 - 2**32 + 1
words = lambda *s: g.integers(0, P, size=s, dtype=np.uint64)
h = hashlib.sha256()
def put(pf):
    for a in (pf.round_polys, pf.challenges, pf.final_value):
        h.update(np.ascontiguousarray(a).tobytes())
K = lambda f=3: E.Transcript.keccak(f, b"pdl")
n = 17
for cls in (E.InnerProductProver, E.InnerProductProverLSB):
    tabs = [words(1 << n) for _ in range(2)]
    for p in (cls(*tabs), cls.from_host(tabs)):
        for graph in (True, False):
            put(p.prove(n, K(), use_graph=graph)); p.reset()
for cls in (E.MultilinearProver, E.MultilinearProverLSB):
    t = words(1 << 18)
    put(cls(t).prove(18, K())); put(cls(t, field=1).prove(12, K(1)))
put(E.InnerProductProver(words(40001), words(40001)).prove(16, K()))
for cls in (E.CoefficientProver, E.CoefficientProverLSB):
    put(cls([words(1 << 14, 3), words(1 << 14), words(1 << 14)]).prove(14, K(), hook=b"abc"))
put(E.EqFactoredProver(words(17, 3), words(1 << 17)).prove(17, K()))
put(E.GkrProver(words(1 << 12), words(1 << 12), words(64)).prove(12, K()))
for width, count, field in ((8, 1 << 12, 1), (3, 1 << 9, 3), (700, 33, 1), (9000, 5, 3)):
    levels = count.bit_length() - 1
    pairs = [(words(field), words(field)) for _ in range(levels)]
    polys = words(count, width) if field == 1 else words(count, width, 3)
    h.update(np.ascontiguousarray(E.protogalaxy_fold(pairs, polys, field=field)).tobytes())
print(h.hexdigest())
"""


@pytest.mark.gpu
def test_every_launch_form_gives_the_same_words():
    got = {}
    for form in (None, "0", "1"):
        env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "efficient-sumcheck_gb300"))
        env.pop("EFFSC_PDL", None)
        if form is not None:
            env["EFFSC_PDL"] = form
        r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got[form] = r.stdout.strip()
    assert len(got["0"]) == 64 and got[None] == got["0"] == got["1"]
