"""The FP64 form's two kernels against tuple energies evaluated beyond FP64: W
from exact products of 21-bit parts of the operands, the rest in long double.

The tensor-core kernel must be as accurate as the FP64-instruction kernel: its
2-norm error over the tuples at most 4 times that one's (the two are samples of
the same size of rounding error).  A lost or misplaced level of digit products
is 2^8 and more of it."""
import numpy as np
import pytest

import oracle
from atrip_gb300 import capi, synth

NAMES = ("epsi", "epsa", "Tai", "Tabij", "Vabij", "Vijka", "Vabci")
J2 = ("Jijka", "Jabci")


def _parts(x):
    """x = sum of three parts, whole multiples of 2^(e - 21 (k + 1)) below 2^21 of them."""
    e = np.frexp(np.max(np.abs(x)))[1] if x.size else 0
    out = []
    for k in range(3):
        s = np.ldexp(1.0, int(21 * (k + 1) - e))
        p = np.rint(x * s) / s
        out.append(p)
        x = x - p
    return out


def _matmul(a, b):
    """a @ b (real, at most 1024 terms) to about 2^-80 of the largest product."""
    pa, pb = _parts(a), _parts(b)
    r = np.zeros((a.shape[0], b.shape[1]), dtype=np.longdouble)
    for i in range(3):
        for j in range(3 - i):
            r += (pa[i] @ pb[j]).astype(np.longdouble)  # each exact in FP64
    return r


def _product(a, b):
    if not np.iscomplexobj(a):
        return _matmul(a, b)
    re = _matmul(a.real, b.real) - _matmul(a.imag, b.imag)
    return re + 1j * (_matmul(a.real, b.imag) + _matmul(a.imag, b.real))


def _w(d, vh, vp, a, b, c):
    T, Vh, Vp, No = d["Tabij"], d[vh], d[vp], d["No"]

    def term(x, w, y, z, u, v, flip):
        rows = T[x].transpose(1, 2, 0).reshape(No * No, -1)  # (p,q), E
        hole = Vh[:, :, :, w].reshape(No * No, No).conj()  # (p,q), L
        col = T[u, v].T if flip else T[u, v]  # L, r
        return (_product(rows, Vp[y, z]) - _product(hole, col)).reshape(No, No, No)

    w = term(a, b, b, c, a, c, False)
    w = w + term(a, c, c, b, a, b, False).transpose(0, 2, 1)
    w = w + term(c, a, a, b, b, c, True).transpose(1, 2, 0)
    w = w + term(c, b, b, a, a, c, True).transpose(2, 1, 0)
    w = w + term(b, a, a, c, b, c, False).transpose(1, 0, 2)
    return w + term(b, c, c, a, a, b, True).transpose(2, 0, 1)


def _energies(d, tuples, j):
    """(e, ect) of the tuples, in long double."""
    No, kind = d["No"], np.clongdouble if np.iscomplexobj(d["Tabij"]) else np.longdouble
    I, J, K = np.array([(i, q, k) for k in range(No) for q in range(k, No) for i in range(q, No)]).T
    fac = np.where(J == K, 0.5, 1.0) * np.where(I == J, 0.5, 1.0)
    ei, ea, t1, V = (d[k].astype(kind) for k in ("epsi", "epsa", "Tai", "Vabij"))
    out = []
    for a, b, c in tuples:
        W = _w(d, "Vijka", "Vabci", a, b, c)
        Z = (W + t1[a][:, None, None] * V[b, c][None] + t1[b][None, :, None] * V[a, c][:, None, :] +
             t1[c][None, None, :] * V[a, b][:, :, None])
        den = (ea[a] + ea[b] + ea[c]).real - (ei[I] + ei[J] + ei[K])

        def energy(T):
            def six(X):
                return [X[p, q, r] for p, q, r in ((I, J, K), (I, K, J), (J, I, K), (J, K, I),
                                                   (K, I, J), (K, J, I))]
            U, V2, W2, X, Y, Z2 = six(Z)
            A, B, C, D, E, F = six(T.conj())
            uxy, vwz, ade, bcf = U + X + Y, V2 + W2 + Z2, A + D + E, B + C + F
            first = A * U + B * V2 + C * W2 + D * X + E * Y + F * Z2
            val = 3 * first + (uxy - 2 * vwz) * ade + (vwz - 2 * uxy) * bcf
            if a == b or b == c:
                val = 3 * (A * U + D * X + E * Y) - ade * uxy
            return ((2 * val / den).real * fac).sum()

        e = energy(W)
        out.append((e, energy(_w(d, "Jijka", "Jabci", a, b, c)) if j else e))
    return np.array(out).T


def _tuples(Nv, t0, n):
    return [capi.tuple_at(Nv, t0 + k) for k in range(n)]


# the evaluation itself, against the FP64 oracle
@pytest.mark.parametrize("field", ["real", "complex"])
def test_evaluation_matches_the_oracle(field):
    d = synth.make_inputs(5, 9, 41, with_j=True, field=field, eps_imag=0.05 if field == "complex" else 0.0)
    n = 40
    got = _energies(d, _tuples(9, 0, n), True)
    want = oracle.tuple_energies(oracle.Problem(d), 0, n)
    for x, y in zip(got, want):
        assert np.max(np.abs(x.astype(float) - y)) <= 2 * 14 * 2 * 2.0 ** -52 * np.max(np.abs(y))


# every column count P of the kernel, with slots of two and of four slices, one
# and two accumulators
@pytest.mark.gpu
@pytest.mark.parametrize("No,Nv,j,field", [
    (6, 60, True, "real"), (8, 40, True, "real"), (15, 33, False, "real"), (24, 30, True, "real"),
    (31, 24, False, "real"), (37, 40, True, "real"), (46, 18, False, "real"),
    (56, 14, False, "real"), (63, 12, False, "real"), (24, 160, False, "real"),
    (7, 36, True, "complex"), (13, 26, False, "complex"), (21, 20, True, "complex"),
    (32, 14, False, "complex")])
def test_as_accurate_as_fp64_instructions(No, Nv, j, field):
    d = synth.make_inputs(No, Nv, 42, with_j=j, field=field,
                          eps_imag=0.05 if field == "complex" else 0.0)
    n, t0 = 24 if No <= 32 else 10, synth.n_tuples(Nv) // 3
    kw = dict(form="fp64", use_j=j, first_iteration=t0, max_iterations=t0 + n - 1)
    with capi.Context(No, Nv, 0, field=field) as ctx:
        for k in NAMES + (J2 if j else ()):
            ctx.upload(k, d[k])
        ctx.run(**kw)
        assert ctx.last_kernel() == "tensor_core"
        tc = ctx.tuple_energies(t0, n)
        ctx.set_tuning(fp64_tile_rows=64)
        ctx.run(**kw)
        assert ctx.last_kernel() == "fp64_instructions"
        dfma = ctx.tuple_energies(t0, n)
    want = _energies(d, _tuples(Nv, t0, n), j)
    for x, y, ref in zip(tc, dfma, want):
        err = [float(np.sqrt(np.sum((v.astype(np.longdouble) - ref) ** 2))) for v in (x, y)]
        print(No, Nv, field, "tensor cores %.2e, FP64 instructions %.2e of the 2-norm" %
              tuple(e / float(np.sqrt(np.sum(ref ** 2))) for e in err))
        assert err[0] <= 4 * err[1]


# pair slabs of T that symmetry leaves at round-off: no product of a whole T_x is
# small, so the tensor cores take them
@pytest.mark.gpu
@pytest.mark.parametrize("No,Nv", [(8, 40), (15, 33)])
def test_pair_slabs_at_round_off(No, Nv):
    d = synth.make_inputs(No, Nv, 43)
    u = np.arange(Nv)
    d["Tabij"][(u[:, None] + u[None, :]) % 2 == 1] *= 1e-17
    n, t0 = 24, synth.n_tuples(Nv) // 2
    kw = dict(form="fp64", use_j=False, first_iteration=t0, max_iterations=t0 + n - 1)
    with capi.Context(No, Nv, 0) as ctx:
        for k in NAMES:
            ctx.upload(k, d[k])
        ctx.run(**kw)
        assert ctx.last_kernel() == "tensor_core"
        tc = ctx.tuple_energies(t0, n)[0]
        ctx.set_tuning(fp64_tile_rows=64)
        ctx.run(**kw)
        dfma = ctx.tuple_energies(t0, n)[0]
    ref = _energies(d, _tuples(Nv, t0, n), False)[0]
    err = [float(np.sqrt(np.sum((v.astype(np.longdouble) - ref) ** 2))) for v in (tc, dfma)]
    assert err[0] <= 4 * err[1]
