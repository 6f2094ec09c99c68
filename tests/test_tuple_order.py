"""The processing order of a stretch of the tuple list (csrc/tuple_order.cuh)."""
import ctypes
import os
import subprocess
import time

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def block_order(tmp_path_factory):
    d = tmp_path_factory.mktemp("tuple_order")
    src = d / "order.cpp"
    src.write_text('#include "tuple_order.cuh"\n'
                   'extern "C" void order(const uint32_t *t, int64_t n, int nv, int l, uint32_t *o) {\n'
                   '  atrip_gb300::block_order(t, n, nv, l, o);\n}\n')
    lib = d / "order.so"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "atrip_gb300", "csrc"), str(src), "-o", str(lib)])
    fn = ctypes.CDLL(str(lib)).order
    P = ctypes.POINTER(ctypes.c_uint32)

    def call(tuples, nv, side):
        out = np.full(len(tuples) + 1, 0xffffffff, dtype=np.uint32)
        fn(tuples.ctypes.data_as(P), ctypes.c_int64(len(tuples)), nv, side, out.ctypes.data_as(P))
        assert out[-1] == 0xffffffff
        return out[:-1]
    return call


def _list(nv):
    a, b, c = np.meshgrid(*[np.arange(nv, dtype=np.uint32)] * 3, indexing="ij")
    keep = (a <= b) & (b <= c) & ~((a == b) & (b == c))
    return (a | (b << 10) | (c << 20))[keep].astype(np.uint32)


@pytest.mark.parametrize("nv,side", [(2, 2), (9, 2), (10, 4), (23, 4), (40, 6), (40, 7), (40, 64)])
@pytest.mark.parametrize("part", [(0.0, 1.0), (0.3, 0.31), (0.5, 0.9), (0.7, 0.7)])
def test_blocks_in_list_order(block_order, nv, side, part):
    t = _list(nv)
    t = np.ascontiguousarray(t[int(part[0] * len(t)):int(part[1] * len(t))])
    a, b, c = t & 0x3ff, (t >> 10) & 0x3ff, t >> 20
    want = np.lexsort((np.arange(len(t)), c // side, b // side, a // side))
    np.testing.assert_array_equal(block_order(t, nv, side), want)


# a driver that walks the list in short stretches orders each of them: 300 of
# 1000 tuples, seconds with a counter for every one of 256^3 block triples
def test_short_stretches_of_a_long_list(block_order):
    nv = 1023
    rng = np.random.default_rng(0)
    t = np.sort(rng.integers(0, nv, (3, 1000)), axis=0).astype(np.uint32)
    t = np.ascontiguousarray(np.sort(t[0] | (t[1] << 10) | (t[2] << 20)))
    t0 = time.perf_counter()
    for _ in range(300):
        block_order(t, nv, 4)
    assert time.perf_counter() - t0 < 0.5
