"""The check behind trips_debug_lists and trips_debug_list_starts (csrc/list_order.h): lists in any order that fill their part of
the list buffer pass, lists that overlap, leave it or leave slots over do not."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def covers(tmp_path_factory):
    d = tmp_path_factory.mktemp("list_order")
    src = d / "cover.cpp"
    src.write_text('#include "list_order.h"\n'
                   'extern "C" int cover(const uint32_t* s, const uint32_t* c, size_t n, uint64_t nf) { return trips::lists_cover(s, c, n, nf); }\n')
    so = d / "cover.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "trips_b200", "csrc"), str(src), "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).cover
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_uint64]

    def call(starts, counts, n_frags):
        s, c = np.asarray(starts, np.uint32), np.asarray(counts, np.uint32)
        return bool(fn(s.ctypes.data, c.ctypes.data, s.size, int(n_frags)))
    return call


def _lists(rng, n=5000):
    """Lists of 0..8 fragments in a shuffled order."""
    counts = rng.integers(0, 9, n)
    starts = np.empty(n, np.int64)
    order = rng.permutation(n)
    starts[order] = np.concatenate([[0], np.cumsum(counts[order])[:-1]])
    return starts, counts


def test_lists_in_any_order(covers):
    starts, counts = _lists(np.random.default_rng(1))
    assert covers(starts, counts, counts.sum())
    assert covers([], [], 0) and covers([7, 0], [0, 0], 0)


@pytest.mark.parametrize("fault", ["overlap", "gap", "beyond", "wrapped", "missing", "same_range"])
def test_misplaced_lists(covers, fault):
    starts, counts = _lists(np.random.default_rng(2))
    n_frags = int(counts.sum())
    k = int(np.flatnonzero((counts > 1) & (starts > 0))[0])
    if fault == "overlap":
        starts[k] -= 1
    elif fault == "gap":
        starts[starts >= starts[k]] += 1
    elif fault == "beyond":
        starts[k] = n_frags - counts[k] + 1
    elif fault == "wrapped":  # an end before its length: the collect pass did not finish the list
        starts[k] = 2**32 - 1
    elif fault == "missing":
        counts[k] = 0
    elif fault == "same_range":
        j = int(np.flatnonzero((counts == counts[k]) & (np.arange(counts.size) != k))[0])
        starts[k] = starts[j]
    assert not covers(starts, counts, n_frags)
