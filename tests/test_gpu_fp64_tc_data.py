"""Data the FP64 form's digit slices would hold less exactly than FP64 does
runs on the FP64-instruction kernels, with their results."""
import ctypes

import numpy as np
import pytest

from atrip_gb300 import capi, synth

pytestmark = pytest.mark.gpu
NAMES = ("epsi", "epsa", "Tai", "Tabij", "Vabij", "Vijka", "Vabci")
J2 = ("Jijka", "Jabci")


def _ctx(d, j=False, field="real"):
    ctx = capi.Context(d["No"], d["Nv"], 0, field=field)
    for n in NAMES + (J2 if j else ()):
        ctx.upload(n, d[n])
    return ctx


def _decoupled(No, Nv, bits, j=False, field="real", zero_x=False):
    """Amplitudes that vanish for two core orbitals and half the virtuals E;
    the integrals that meet the others 2^-bits of those that meet none.  Slab
    maxima all lie within a few bits of the tensors'.  j: the (cT)
    intermediates are so, V is not."""
    d = synth.make_inputs(No, Nv, 21, with_j=j, field=field)
    h = Nv // 2
    T = d["Tabij"]
    T[:, :, :2] = 0
    T[:, :, :, :2] = 0
    T[:, :h] = 0
    if zero_x:
        T[:h] = 0
    d["Jabci" if j else "Vabci"][:, :, h:] *= 2.0 ** -bits
    return d


def _run(ctx, n, j=False):
    ctx.run(form="fp64", max_iterations=n - 1, use_j=j)
    return ctx.tuple_energies(0, n)


@pytest.mark.parametrize("bits", [8, 20, 30])
@pytest.mark.parametrize("field,j,zero_x", [("real", False, False), ("real", False, True),
                                            ("real", True, False), ("complex", False, False)])
def test_decoupled_operands(bits, field, j, zero_x):
    d = _decoupled(8, 40, bits, j, field, zero_x)
    with _ctx(d, j, field) as ctx:
        e, ect = _run(ctx, 1000, j)
        ctx.set_tuning(fp64_tile_rows=64)
        f, fct = _run(ctx, 1000, j)
    np.testing.assert_array_equal(e, f)
    np.testing.assert_array_equal(ect, fct)


# in a batch: such a system, one whose level sums leave their exact range, and
# one the tensor cores take
def test_decoupled_operands_in_a_batch():
    ds = [_decoupled(8, 40, 20), synth.make_inputs(9, 42, 22), synth.make_inputs(8, 41, 23)]
    ds[1]["Tabij"][:] = 1.0 / 3.0
    ds[1]["Vabci"][:] = 1.0 / 3.0
    ctxs = [_ctx(d) for d in ds]
    n = [synth.n_tuples(d["Nv"]) for d in ds]
    with capi.Batch(ctxs) as b:
        b.run(form="fp64", use_j=False)
        e = [c.tuple_energies(0, m)[0] for c, m in zip(ctxs, n)]
        b.set_tuning(tuples_per_claim=1)  # the batch kernel of FP64 instructions
        b.run(form="fp64", use_j=False)
        f = [c.tuple_energies(0, m)[0] for c, m in zip(ctxs, n)]
    np.testing.assert_array_equal(e[0], f[0])
    np.testing.assert_array_equal(e[1], f[1])
    assert np.max(np.abs(e[2] - f[2])) <= 2 * 49 * 2.0 ** -52 * np.max(np.abs(f[2]))
    for c in ctxs:
        c.close()
