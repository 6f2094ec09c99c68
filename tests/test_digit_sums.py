"""The rule by which the FP64 form's level sums are taken to be exact in FP32
accumulators (csrc/digit_sums.cuh), against sums formed in FP32."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SLICES, NORMS = 8, 7


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("digit_sums")
    src = d / "rule.cpp"
    src.write_text('#include "digit_sums.cuh"\n'
                   'extern "C" int rule(int terms, const double *n, int loose) {\n'
                   '  const auto *x = reinterpret_cast<const atrip_gb300::DigitNorms *>(n);\n'
                   '  return atrip_gb300::level_sums_exact(terms, x[0], x[1], x[2], x[3], loose != 0);\n'
                   '}\n')
    lib = d / "rule.so"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "atrip_gb300", "csrc"), str(src), "-o", str(lib)])
    fn = ctypes.CDLL(str(lib)).rule

    def call(terms, norms, loose=False):
        a = np.ascontiguousarray(norms, dtype=np.float64)
        assert a.shape == (4, NORMS)
        return bool(fn(terms, a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), int(loose)))
    return call


def _level_sums(q, r, level):
    """(FP32, exact) sum over k of the level's digit products, k by k."""
    t = sum(q[s] * r[level - s] for s in range(level + 1))  # whole numbers
    acc = np.float32(0)
    for x in t:
        acc = np.float32(acc + np.float32(x))
    return float(acc), float(t.sum())


# operands whose digit products have one sign along the natural half of K and
# the other along the transposed half: every level's sum runs up and comes back
# to nearly zero, so its end shows nothing
@pytest.mark.parametrize("top", [(118, 62, 46), (126, 30, 20), (100, 90, 40), (64, 1, 1)])
@pytest.mark.parametrize("nv", [100, 180, 240, 400, 560])
def test_accepted_sums_are_exact(rule, top, nv):
    rng = np.random.default_rng(nv)
    q = np.array(list(top) + [127] * (SLICES - 3), dtype=np.int64)[:, None] * np.ones((1, nv), np.int64)
    r = q.copy()
    r[3:] -= rng.integers(0, 2, (SLICES - 3, nv))  # odd and even products
    n = [[float((x[s] ** 2).sum()) for s in range(NORMS)] for x in (q, r)]
    zero = [0.0] * NORMS
    rows, cols = np.concatenate([q, q], 1), np.concatenate([r, -r], 1)
    half = [_level_sums(q, r, L) for L in range(NORMS)]
    both = [_level_sums(rows, cols, L) for L in range(NORMS)]
    assert all(abs(y) < 2 ** 22 for _, y in both)
    if rule(2, [n[0], n[1], zero, zero]):
        assert all(x == y for x, y in both)
    if rule(1, [n[0], n[1], zero, zero]):
        # a half alone: exact where its end lies within what is checked
        assert all(x == y for x, y in half if abs(y) < 2 ** 22)
    if rule(2, [n[0], n[1], zero, zero], loose=True):
        assert all(x == y for x, y in both[:6])
        assert abs(both[6][0] - both[6][1]) <= 2 * 7 * 2 * nv  # 2 for each product
    exact = all(x == y for x, y in both)
    assert exact or not rule(2, [n[0], n[1], zero, zero])


# operands that only the loose rule accepts: level 6 passes 2^24 and is rounded
def test_loose_level_six(rule):
    nv = 560
    rng = np.random.default_rng(1)
    q = np.array([64, 1, 1] + [127] * 5, dtype=np.int64)[:, None] * np.ones((1, nv), np.int64)
    r = q.copy()
    r[1:] -= rng.integers(0, 2, (SLICES - 1, nv))
    n = [[float((x[s] ** 2).sum()) for s in range(NORMS)] for x in (q, r)] + [[0.0] * NORMS] * 2
    assert not rule(2, n) and rule(2, n, loose=True)
    rows, cols = np.concatenate([q, q], 1), np.concatenate([r, -r], 1)
    for L in range(NORMS):
        x, y = _level_sums(rows, cols, L)
        assert x == y if L < 6 else abs(x - y) <= 2 * 7 * 2 * nv


# normal operands: one accumulator up to Nv + No ~ 360 (loose 450), two (one per
# half) up to the longest K the form serves
@pytest.mark.parametrize("no,nv,terms", [(8, 40, 2), (24, 240, 2), (42, 240, 2), (37, 151, 2),
                                         (56, 440, 1), (30, 660, 1)])
def test_normal_operands_are_accepted(rule, no, nv, terms):
    rng = np.random.default_rng(no)

    def norms(k, rows):
        x = rng.normal(size=(rows, k))
        y = np.rint(x * (126 / np.abs(x).max() * 0.6) * 2.0 ** 40).astype(np.int64)
        out = []
        for s in range(6):  # balanced digits from the bottom up
            d = (y + 128) % 256 - 128
            out.append(float((d * d).sum(1).max()))
            y = (y - d) >> 8
        return out[::-1] + [out[0]]  # digit 6 like digit 5
    n = [norms(nv, 4000), norms(nv, 4000), norms(no, 4000), norms(no, 4000)]
    assert rule(terms, n) and rule(terms, n, loose=True)
    if terms == 1:
        assert not rule(2, n)


def test_normal_operands_loose(rule):
    rng = np.random.default_rng(7)

    def norms(k):
        x = rng.normal(size=(4000, k))
        y = np.rint(x * (126 / np.abs(x).max() * 0.6) * 2.0 ** 40).astype(np.int64)
        out = []
        for s in range(6):
            d = (y + 128) % 256 - 128
            out.append(float((d * d).sum(1).max()))
            y = (y - d) >> 8
        return out[::-1] + [out[0]]
    n = [norms(400), norms(400), norms(40), norms(40)]
    assert rule(2, n, loose=True) and not rule(2, n)
