"""How many blocks the tensor-core start of many proofs takes: the server holds
partial sums for tc_blocks_most of them from its creation on and allocates
nothing in a step, so no mix of requests that its budget admits may need more.
The rule is compiled for the host; no GPU."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "efficient-sumcheck_gb300", "csrc")

# in: sms, budget, proofs, their variables; out: tiles a block, the blocks of
# the launch, the most the budget and the number of proofs allow
HARNESS = r"""
#include <cstdio>
#include "tc_plan.h"
using namespace effsc;
int main() {
    unsigned long long sms, budget, most_active, n;
    while (std::scanf("%llu %llu %llu %llu", &sms, &budget, &most_active, &n) == 4) {
        unsigned long long nv[4096], total = 0, blocks = 0;
        for (unsigned long long i = 0; i < n; i++) { std::scanf("%llu", nv + i); total += (1ull << (nv[i] - 4)) / 128; }
        const unsigned long long per = tc_tiles_per_block(total, sms, 512);
        for (unsigned long long i = 0; i < n; i++) blocks += ((1ull << (nv[i] - 4)) / 128 + per - 1) / per;
        std::printf("%llu %llu %llu\n", per, blocks, (unsigned long long)tc_blocks_most(budget / (40 * 16 * 128), most_active, sms, 512));
    }
}
"""


def test_blocks_fit(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(HARNESS)
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)])
    rng = random.Random(4)
    lines = []
    for budget in (1 << 20, 1 << 30, 8 << 30, 64 << 30, 280 << 30):
        for active in (1, 3, 64, 4096):
            for sms in (132, 152):
                for top in (14, 18, 22, 26, 33):
                    left, nv = budget, []
                    while len(nv) < active and left >= 40 << 14:      # as the admission does
                        v = rng.randint(14, top)
                        while 40 << v > left:
                            v -= 1
                        left -= 40 << v
                        nv.append(v)
                    if nv:
                        lines.append("%d %d %d %d %s" % (sms, budget, active, len(nv), " ".join(map(str, nv))))
    out = subprocess.run([str(exe)], input="\n".join(lines), capture_output=True, text=True, check=True).stdout.split("\n")
    for line, got in zip(lines, out):
        per, blocks, most = map(int, got.split())
        assert 16 <= per <= 512 and 0 < blocks <= most, (line[:80], got)
    assert len(out) == len(lines) + 1


def test_partials_hold_every_pass(tmp_path):
    """The words that each kind's passes write, from the kernels' sources, fit."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text("""#include <cstdio>
#include "tc_plan.h"
int main() { for (int s = 1; s <= 200; s++) std::printf("%zu %zu %zu\\n", effsc::partial_words(true, false, 8 * s), effsc::partial_words(false, true, 8 * s),
    effsc::partial_words(false, false, 8 * s)); }""")
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)])
    rows = [[int(x) for x in r.split()] for r in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split("\n") if r]
    assert len(rows) == 200
    for sms, (ip, coef, other) in enumerate(rows, 1):
        rounds = 8 * sms * 12                        # round_common.cuh: RAW_WORDS a block
        # k_ip_gram: 16 x 16 words a block, one an SM; ip012.cuh: 32, two an SM
        assert ip >= max(rounds, sms * 256, 2 * sms * 32)
        # k_c3_gram: 12 x 9, one an SM; coef01.cuh: 48, a quarter of the grid
        assert coef >= max(rounds, sms * 108, 2 * sms * 48)
        assert other == rounds


@pytest.mark.gpu
def test_small_provers_stay_small():
    """What a prover without tables of a size holds on the device."""
    import ctypes
    import numpy as np
    import effsc_gpu as E
    E.MultilinearProver(np.arange(8, dtype=np.uint64))
    rt = ctypes.CDLL("libcudart.so.13")
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0

    def now():
        E.Context.default().synchronize()
        assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0       # cudaMemPoolAttrUsedMemCurrent
        return used.value
    at = now()
    keep = [E.MultilinearProver(np.arange(8, dtype=np.uint64)) for _ in range(32)]
    assert now() - at < 32 * (200 << 10)
    del keep


def test_a_step_allocates_nothing():
    text = open(os.path.join(CSRC, "serve.cu")).read()
    body = text[text.index("\nint step("):]
    body = body[:body.index("\n}")]
    assert "Malloc" not in body and "HostAlloc" not in body
