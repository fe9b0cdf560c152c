"""Where a table is decides how passes read it in place: those whose waits have
the usual time limit take device and pinned memory alone, since a pageable (or
managed) page may first have to be brought in.  The rules are compiled for the
host and checked without a GPU; on the GPU, tables of each kind are proved, and
with that limit at zero, which only a pass without such waits survives."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "efficient-sumcheck_gb300", "csrc")

HARNESS = r"""
#include <cstdio>
#include <initializer_list>
#include <vector>
#include <sys/mman.h>
#include "residency.h"
using namespace effsc;
static size_t resident(void* p, size_t bytes) {
    const size_t page = sysconf(_SC_PAGESIZE);
    std::vector<unsigned char> v(bytes / page);
    if (mincore(p, bytes, v.data())) return 0;
    size_t n = 0;
    for (unsigned char x : v) n += x & 1;
    return n;
}
int main() {
    for (Residency r : {Residency::device, Residency::managed, Residency::pinned, Residency::pageable})
        std::printf("%d ", (int)prompt_reads(r));
    std::printf("%llu %llu ", (unsigned long long)tc_wait_ns(false), (unsigned long long)tc_wait_ns(true));
    // untouched memory: from the second page's fourth word to the fourth page's
    const size_t page = sysconf(_SC_PAGESIZE);
    char* m = (char*)mmap(nullptr, 8 * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    touch_pages(m + page + 24, 2 * page);
    std::printf("%d %d ", (int)resident(m + page, 3 * page), (int)resident(m, 8 * page));
    munmap(m + 4 * page, 4 * page);
    touch_pages(m, 4 * page);              // the next page is a hole
    touch_pages(m + 4 * page, 0);
    std::printf("%d ", (int)resident(m, 4 * page));
    unsigned long long L, rounds, addr, prompt, copied;
    while (std::scanf("%llu %llu %llu %llu %llu", &L, &rounds, &addr, &prompt, &copied) == 5)
        std::printf("%d ", ip_start_rounds(L, rounds, addr, prompt != 0, copied != 0, 128));
}
"""


def test_rules(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(HARNESS)
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)])
    cases, want = [], []
    for lg in range(14, 40):
        for rounds in (4, 5, lg):
            for addr in (0, 16, 8, 24):
                for prompt in (0, 1):
                    for copied in (0, 1):
                        nv = 4 if rounds >= 5 else 3
                        tiles = (1 << lg) // (1 << nv) // 128
                        cases.append("%d %d %d %d %d" % (1 << lg, rounds, addr, prompt, copied))
                        want.append(nv if (prompt or copied) and addr % 16 == 0 and 1 <= tiles < 1 << 31 else 0)
    out = subprocess.run([str(exe)], input="\n".join(cases), capture_output=True, text=True, check=True).stdout.split()
    out = [int(x) for x in out]
    assert out[:4] == [1, 0, 1, 0]                            # device, managed, pinned, pageable
    assert out[4] == 10**9 and out[5] >= 3200 * 30 * 10**6    # every page in flight at a slow disk's pace
    assert out[6:9] == [3, 3, 4]                              # the pages of the range, and no others
    assert out[9:] == want


HARNESS_COPY = r"""
#include <cstdio>
#include "residency.h"
using namespace effsc;
static int waits = 0;
static int leave(int at, bool in_place) {     // a scope with three ways out
    ReadsInPlace reads([] { waits++; return at_error; });
    if (at == 0) return 10;
    reads.pending |= in_place;
    if (at == 1) return 11;                    // an error after the reads began
    if (reads.finish()) return 12;
    return 0;
}
int main() {
    for (int in_place = 0; in_place < 2; in_place++)
        for (int at = 0; at < 3; at++) {
            waits = 0;
            const int rc = leave(at, in_place);
            std::printf("%d %d ", rc, waits);
        }
    at_error = 7;
    waits = 0;
    const int rc = leave(2, true);
    std::printf("%d %d ", rc, waits);
    const Residency all[4] = {Residency::device, Residency::managed, Residency::pinned, Residency::pageable};
    for (Residency r : all)
        for (int tables = 0; tables < 2; tables++)
            for (size_t words : {(size_t)8191, (size_t)8192})
                for (uintptr_t address : {(uintptr_t)4096, (uintptr_t)4100})
                    std::printf("%d", (int)kernel_copies(r, tables != 0, words, address));
}
"""


def test_copies_in_place(tmp_path):
    """Who copies by a kernel, and that a scope with reads in flight is never left
    before they are done: not by an error's way out, not twice, not for nothing."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "c.cpp", tmp_path / "c"
    src.write_text("#include <initializer_list>\nstatic int at_error = 0;\n" + HARNESS_COPY)
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    assert [int(x) for x in out[:14]] == [10, 0, 11, 0, 0, 0, 10, 0, 11, 1, 0, 1, 12, 1]
    assert out[14] == "0" * 30 + "10"          # pageable, host page tables, 64 KB, aligned
    serve = open(os.path.join(CSRC, "serve.cu")).read()
    body = serve[serve.index("int admit("):]
    body = body[:body.index("\n}")]
    assert body.index("ReadsInPlace reads(") < body.index("TRYS(") and "&reads.pending" in body


@pytest.fixture(scope="module")
def E():
    import effsc_gpu
    effsc_gpu.load()
    O.set_threads(os.cpu_count() or 1)
    return effsc_gpu


@pytest.fixture()
def place():
    """place(kind, arrays): the arrays' words in memory of that kind, as pointers."""
    keep = []

    def put(kind, arrays):
        out = []
        for a in arrays:
            a = np.ascontiguousarray(a)
            if kind == "managed":
                rt = ctypes.CDLL("libcudart.so.13")
                p = ctypes.c_void_p()
                assert rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(a.nbytes), ctypes.c_uint(1)) == 0
                ctypes.memmove(p, a.ctypes.data, a.nbytes)
                keep.append(lambda p=p: rt.cudaFree(p))
                out.append(p.value)
            else:
                import torch
                t = torch.from_numpy(a.view(np.int64)).pin_memory() if kind == "pinned" else a
                keep.append(lambda t=t: None)
                out.append(t.numpy().view(np.uint64) if kind == "pinned" else t)
        return out
    yield put
    for free in keep:
        free()


def tables(kind, n):
    g = np.random.default_rng(n)
    return [g.integers(0, O.P, size=1 << n, dtype=np.uint64) for _ in range({"ip": 2, "ml": 1, "coef": 3}[kind])]


def proof_is(pf, kind, lsb, tabs, rounds):
    rp, ch, fv = O.sumcheck(O.Prover({"ip": O.IP, "ml": O.ML, "coef": O.COEF}[kind], O.LSB if lsb else O.MSB, 3, tabs), rounds,
                            O.Transcript(3, label=b"res"))
    return (np.array_equal(pf.round_polys, rp[:, :pf.round_polys.shape[1]]) and np.array_equal(pf.challenges, ch)
            and np.array_equal(pf.final_value, fv))


@pytest.mark.gpu
@pytest.mark.parametrize("lsb", [False, True])
@pytest.mark.parametrize("kind", ["resident", "mapped file", "untouched"])
def test_pageable_tables(E, lsb, kind, tmp_path):
    """Pages that are there, that a new mapping has not met, and that nothing has
    touched (zeros); with fewer rounds too."""
    n = 19
    tabs = tables("ip", n)
    if kind == "untouched":
        tabs[0][:] = 0
    cls = E.InnerProductProverLSB if lsb else E.InnerProductProver
    for rounds in (n, 4):
        if kind == "mapped file":
            for i, t in enumerate(tabs):
                t.tofile(str(tmp_path / ("t%d" % i)))
            host = [np.memmap(str(tmp_path / ("t%d" % i)), dtype=np.uint64, mode="r") for i in range(2)]
        else:
            host = [np.zeros(1 << n, dtype=np.uint64) if kind == "untouched" and i == 0 else t for i, t in enumerate(tabs)]
        p = cls.from_host(host, field=3)
        for graph in (False, True):
            assert proof_is(p.prove(rounds, E.Transcript.keccak(3, b"res"), use_graph=graph), "ip", lsb, tabs, rounds)
            p.reset()


@pytest.mark.gpu
@pytest.mark.parametrize("lsb", [False, True])
def test_pinned_tables_take_the_tensor_cores(E, place, lsb):
    tabs = tables("ip", 21)
    cls = E.InnerProductProverLSB if lsb else E.InnerProductProver
    p = cls.from_host(place("pinned", tabs), field=3)
    E.api.check(E.load().effsc_diag_prover_no_wait(p.h, 1))
    with pytest.raises(E.EffscError):
        p.prove(21, E.Transcript.keccak(3, b"res"), use_graph=False)
    E.api.check(E.load().effsc_diag_prover_no_wait(p.h, 0))
    p.reset()
    assert proof_is(p.prove(21, E.Transcript.keccak(3, b"res"), use_graph=False), "ip", lsb, tabs, 21)


@pytest.mark.gpu
@pytest.mark.parametrize("lsb", [False, True])
@pytest.mark.parametrize("kind,n", [("ip", 18), ("ml", 21), ("coef", 16)])
def test_managed_tables_meet_no_time_limit(E, place, kind, n, lsb):
    tabs = tables(kind, n)
    cls = {"ip": (E.InnerProductProver, E.InnerProductProverLSB), "ml": (E.MultilinearProver, E.MultilinearProverLSB),
           "coef": (E.CoefficientProver, E.CoefficientProverLSB)}[kind][lsb]
    p = cls.from_device(place("managed", tabs), [1 << n] * len(tabs), [1] * len(tabs))
    E.api.check(E.load().effsc_diag_prover_no_wait(p.h, 1))
    for graph in (False, True):
        assert proof_is(p.prove(n, E.Transcript.keccak(3, b"res"), use_graph=graph), kind, lsb, tabs, n)
        p.reset()
    del p
