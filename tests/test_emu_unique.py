"""The merge sort of the sorted unique on the CPU, compiled from the kernel source against tests/emu/simt_emu.h: the
positions it leaves are a permutation whatever the ids, also ids wider than key_bits."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "emu", "emu_unique.cpp")
OUT = os.path.join(HERE, "emu", "build", "libemu_unique.so")


@pytest.fixture(scope="module")
def emu():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    deps = [SRC, os.path.join(HERE, "emu", "simt_emu.h"), os.path.join(ROOT, "recsdk_b200", "csrc", "prims.cuh"),
            os.path.join(ROOT, "recsdk_b200", "csrc", "common.cuh"), os.path.join(ROOT, "include", "recsdk_b200.h")]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        subprocess.check_call(["g++", "-O1", "-std=c++17", "-pthread", "-fPIC", "-shared", "-w",
                               f"-I{os.path.join(ROOT, 'include')}", f"-I{os.path.join(ROOT, 'recsdk_b200', 'csrc')}",
                               "-o", OUT, SRC])
    lib = C.CDLL(OUT)
    lib.emu_merge_sort.restype = None
    lib.emu_merge_sort.argtypes = [C.c_void_p, C.c_int64, C.c_int, C.c_void_p]
    lib.emu_merge_sort_pays.restype = C.c_int
    lib.emu_merge_sort_pays.argtypes = [C.c_int64, C.c_int]
    return lib


# sizes at which one of the two sorts took at least a tenth less time than the other
@pytest.mark.parametrize("n,key_bits,merge", [
    (1, 64, 0), (2_048, 20, 0), (2_048, 21, 1), (32_768, 21, 1), (131_072, 21, 0), (196_608, 32, 0), (98_304, 32, 1),
    (131_072, 48, 1), (262_144, 40, 0), (196_608, 64, 1), (131_072, 62, 1), (262_144, 30, 0),
    (524_288, 64, 0), (1 << 20, 21, 0), (1 << 20, 64, 0)])
def test_the_faster_sort_is_taken(emu, n, key_bits, merge):
    assert emu.emu_merge_sort_pays(n, key_bits) == merge


def sorted_bits(key_bits):
    """Bits the radix sort orders by: the fewest passes of 8, 9 or 10 bits, the smallest digit among equals."""
    passes, digit = min((-(-key_bits // d), d) for d in (8, 9, 10))
    return min(passes * digit, 32 if key_bits <= 32 else 64)


# two tiles and one round of merging, or five and two rounds.  Ids of up to id_bits bits, -1 among them.
@pytest.mark.parametrize("key_bits,id_bits,n", [(21, 21, 2_300), (21, 31, 2_300), (21, 31, 8_300), (25, 31, 2_300),
                                                (33, 44, 2_300), (47, 50, 2_300), (64, 63, 2_300)])
def test_merge_sort_is_the_stable_sort_by_the_sorted_bits(emu, key_bits, id_bits, n):
    rng = np.random.default_rng(n + key_bits)
    ids = np.where(rng.random(n) < 0.7, rng.integers(0, 1 << id_bits, n), rng.integers(0, 40, n)).astype(np.int64)
    ids[rng.integers(0, n, 5)] = -1
    order = np.empty(n, np.uint32)
    emu.emu_merge_sort(ids.ctypes.data, n, key_bits, order.ctypes.data)
    np.testing.assert_array_equal(np.sort(order), np.arange(n))
    key = ids.view(np.uint64) & np.uint64((1 << sorted_bits(key_bits)) - 1)
    np.testing.assert_array_equal(order, np.argsort(key, kind="stable"))
