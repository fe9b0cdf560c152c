"""The words that sumcheck_verify_batch hands to the library: each proof's
round polynomials row by row, whatever the memory layout of its array.  The
library is replaced by a recorder, so this runs without a GPU; the values
themselves are checked in test_verify_batch.py."""
import ctypes

import numpy as np
import pytest


@pytest.fixture()
def words(monkeypatch):
    """run(polys) -> the polynomial words that the C call receives."""
    import effsc_gpu.api as A

    class Lib:
        def effsc_verify_batch(self, ctx, field, n, claims, degree, rounds, tx, hook, hook_len, polys, chals, fins):
            total = int(np.frombuffer((ctypes.c_uint32 * n).from_address(ctypes.addressof(rounds)), np.uint32).sum())
            count = total * max(degree, 1) * field
            at = ctypes.cast(polys, ctypes.c_void_p).value
            self.got = np.frombuffer((ctypes.c_uint64 * count).from_address(at), np.uint64).copy()
            return 0

    class Handle:
        h = None

    lib = Lib()
    monkeypatch.setattr(A, "load", lambda: lib)

    def run(polys, degree, field):
        n = len(polys)
        A.sumcheck_verify_batch(np.zeros((n, field), np.uint64), degree, polys, [Handle()] * n, field=field, ctx=Handle())
        return lib.got
    return run


def layouts(a):
    """The same (rounds, degree, field) values in other memory layouts."""
    big = np.zeros((2 * a.shape[0], a.shape[1], 2 * a.shape[2]), a.dtype)
    big[::2, :, ::2] = a
    return {
        "c": a,
        "fortran": np.asfortranarray(a),
        "component-major": np.ascontiguousarray(a.transpose(2, 0, 1)).transpose(1, 2, 0),
        "degree-major": np.ascontiguousarray(a.transpose(1, 0, 2)).transpose(1, 0, 2),
        "strided": big[::2, :, ::2],
        "reversed": np.ascontiguousarray(a[::-1])[::-1],
        "read-only": np.frombuffer(a.tobytes(), a.dtype).reshape(a.shape),
        "int64": a.astype(np.int64),
    }


@pytest.mark.parametrize("layout", ["c", "fortran", "component-major", "degree-major", "strided", "reversed", "read-only",
                                    "int64"])
@pytest.mark.parametrize("rounds", [(2, 2), (5, 1, 0, 7), (3,), (1,)])
def test_words_are_the_rows(words, layout, rounds):
    polys, at = [], 12
    for r in rounds:
        polys.append(np.arange(at, at + r * 6, dtype=np.uint64).reshape(r, 2, 3))
        at += r * 6
    assert np.array_equal(words([layouts(p)[layout] for p in polys], 2, 3), np.arange(12, at, dtype=np.uint64))


def test_mixed_layouts_and_lists(words):
    a = np.arange(24, dtype=np.uint64).reshape(4, 2, 3)
    got = words([np.asfortranarray(a), a.tolist(), a, a.reshape(4, 6)], 2, 3)
    assert np.array_equal(got, np.tile(np.arange(24, dtype=np.uint64), 4))


def test_a_pointer_needs_contiguous_words():
    import effsc_gpu.api as A
    a = np.arange(12, dtype=np.uint64).reshape(3, 4)
    for bad in (a.T, a[:, ::2], np.asfortranarray(a)):
        with pytest.raises(ValueError):
            A._p(bad)
    ro = a.copy()
    ro.flags.writeable = False
    assert np.frombuffer((ctypes.c_uint64 * 12).from_address(ctypes.cast(A._p(ro), ctypes.c_void_p).value), np.uint64)[7] == 7
