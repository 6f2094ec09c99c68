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
        assert ctx.last_kernel() == "fp64_instructions"
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
        assert [c.last_kernel() for c in ctxs] == ["fp64_instructions"] * 2 + ["tensor_core"]
        b.set_tuning(tuples_per_claim=1)  # the batch kernel of FP64 instructions
        b.run(form="fp64", use_j=False)
        f = [c.tuple_energies(0, m)[0] for c, m in zip(ctxs, n)]
    np.testing.assert_array_equal(e[0], f[0])
    np.testing.assert_array_equal(e[1], f[1])
    assert np.max(np.abs(e[2] - f[2])) <= 2 * 49 * 2.0 ** -52 * np.max(np.abs(f[2]))
    for c in ctxs:
        c.close()


# the no-allocation entry point: its FP64-instruction kernel adds in another
# order, so a W cell differs by K 2^-53 of the products it adds and a tuple's
# energy by twice that, times at most its No^3 / 6 triples where they cancel
@pytest.mark.parametrize("bits", [20, 30])
@pytest.mark.parametrize("j", [False, True])
def test_decoupled_operands_noalloc(bits, j):
    torch = pytest.importorskip("torch")
    No, Nv, n = 8, 40, 3000
    d = _decoupled(No, Nv, bits, j)
    names = NAMES + (J2 if j else ())
    dev = {k: torch.from_numpy(np.ascontiguousarray(d[k].ravel(order="F"))).cuda() for k in names}
    out = torch.empty(2 * n + 2, dtype=torch.float64, device="cuda")
    ptrs = capi.DeviceInputs(*[dev[k].data_ptr() if k in dev else None for k in NAMES + J2])
    lib = capi.load()
    torch.cuda.synchronize()
    capi.check(lib.atrip_gpu_run_fp64_noalloc(
        No, Nv, ctypes.byref(ptrs), 0, n - 1, 0, 1, out.data_ptr() + 16,
        out.data_ptr() + 16 + 8 * n, out.data_ptr(), None))
    torch.cuda.synchronize()
    got = out.cpu().numpy()[2:].reshape(2, n)
    with _ctx(d, j) as ctx:
        ctx.set_tuning(fp64_tile_rows=64)
        want = _run(ctx, n, j)
    tol = No ** 3 / 6 * 2 * 2 * (Nv + No) * 2.0 ** -53
    for x, y in zip(got, want):
        assert np.all(np.abs(x - y) <= tol * np.abs(y))


# digits of full size and random signs: the norms of their level sums allow one
# accumulator only up to Nv + No ~ 150 (complex 75), two here
def _digits(rng, shape):
    x = 126.0 * rng.choice([-1.0, 1.0], size=shape)
    for s in range(1, 6):
        x += 127.0 * 2.0 ** (-8 * s) * rng.choice([-1.0, 1.0], size=shape)
    return x * 2.0 ** -7


@pytest.mark.parametrize("No,Nv,j,field", [(4, 160, False, "real"), (5, 155, True, "real"),
                                           (40, 115, False, "real"), (9, 70, False, "complex")])
def test_sums_in_two_accumulators(No, Nv, j, field):
    d = synth.make_inputs(No, Nv, 24, with_j=j, field=field)
    rng = np.random.default_rng(No)
    for k in ("Tabij", "Vijka", "Vabci") + (J2 if j else ()):
        x = _digits(rng, d[k].shape)
        d[k] = x + 1j * _digits(rng, d[k].shape) if field == "complex" else x
    n = 300
    with _ctx(d, j, field) as ctx:
        e, ect = _run(ctx, n, j)
        assert ctx.last_kernel() == "tensor_core"
        ctx.set_tuning(fp64_tile_rows=64)
        f, fct = _run(ctx, n, j)
    K = 2 * (Nv + No) * (2 if field == "complex" else 1)
    assert np.max(np.abs(e - f)) <= K * 2.0 ** -52 * np.max(np.abs(f))
    assert np.max(np.abs(ect - fct)) <= K * 2.0 ** -52 * np.max(np.abs(fct))


# T = 1, V = 1 but for one T_x, or one V_yz, of 2^-bits: the grids' largest
# product is 4, so 4 bits are within 2^6 of it and 5 are not, wherever they are
@pytest.mark.parametrize("bits,kernel", [(4, "tensor_core"), (5, "fp64_instructions")])
@pytest.mark.parametrize("No,Nv", [(8, 40), (8, 41), (9, 39)])
@pytest.mark.parametrize("at", [(0, 1), (-1, -2), (-1, -1), (17, 3), (0,), (33,), (-1,)])
def test_least_product_is_found(bits, kernel, No, Nv, at):
    d = synth.make_inputs(No, Nv, 25)
    d["Tabij"][:] = 1.0
    d["Vabci"][:] = 1.0
    d["Vijka"][:] = 0.5
    if len(at) == 2:
        d["Vabci"][at] = 2.0 ** -bits
        d["Vabci"][at][Nv // 2, No - 1] = 2.0 ** -bits
    else:
        d["Tabij"][at[0]] = 2.0 ** -bits
    with _ctx(d) as ctx:
        ctx.run(form="fp64", use_j=False, max_iterations=9)
        assert ctx.last_kernel() == kernel
