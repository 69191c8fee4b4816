"""The order in which a bead's collision events are folded (fs_events.cuh), compiled for the host:
the places must be a permutation also where keys are equal, or the fold reads list entries that
were never written. Equal keys come from a bead that meets itself where an axis has one cell
(key (cell, position, slot, position), once as i and once as j), and from positions of 4,096 and
more in one cell."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def place(tmp_path_factory):
    d = tmp_path_factory.mktemp("events")
    src = d / "events.cpp"
    src.write_text('#define __host__\n#define __device__\n#define __forceinline__ inline\n#include "fs_events.cuh"\n'
                   'extern "C" void places(const unsigned long long *key, int n, int *out) {\n'
                   '  for (int e = 0; e < n; ++e) out[e] = event_place(key, n, e);\n}\n')
    so = str(d / "events.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "filsim_b200", "csrc"), "-o", so,
                    str(src)], check=True)
    lib = ctypes.CDLL(so)

    def run(key):
        key = np.ascontiguousarray(key, np.uint64)
        out = np.full(len(key), -1, np.int32)
        lib.places(key.ctypes.data_as(ctypes.c_void_p), len(key), out.ctypes.data_as(ctypes.c_void_p))
        return out
    return run


def key(cell, pos_i, slot, pos_j):
    return ((cell * 4096 + pos_i) * 16 + slot) * 4096 + pos_j


def check(place, keys):
    p = place(keys)
    assert sorted(p) == list(range(len(keys)))
    ordered = np.empty(len(keys), np.uint64)
    ordered[p] = keys
    assert np.all(ordered[:-1] <= ordered[1:])


@pytest.mark.parametrize("slots", [[1], [4, 12], list(range(1, 14))])  # one cell along one, two and three axes
def test_a_bead_that_meets_itself(place, slots):
    events = [key(0, 3, s, 3) for s in slots] * 2  # as i, then as j
    events += [key(0, 3, s, 1) for s in [0] + slots] + [key(0, 1, s, 3) for s in slots]
    rng = np.random.default_rng(len(slots))
    for _ in range(20):
        check(place, rng.permutation(np.array(events, np.uint64)))


def test_positions_past_the_key(place):
    # the key of position 4,096 under slot 2 is that of position 0 under slot 3
    check(place, np.array([key(5, 9, 2, 4096), key(5, 9, 3, 0), key(5, 9, 2, 1)], np.uint64))


def test_all_equal_up_to_the_list(place):
    for n in (0, 1, 2, 63, 64):
        check(place, np.full(n, 77, np.uint64))


def test_distinct_keys_sort(place):
    rng = np.random.default_rng(0)
    check(place, rng.permutation(np.array([key(c, i, s, j) for c in (0, 9) for i in (0, 4095) for s in (0, 13)
                                           for j in (0, 2, 4095)], np.uint64)))
