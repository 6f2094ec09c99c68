"""Operands the split forms' tensor-core kernel cannot take as integers, against
the split kernels that a variant selects."""
import numpy as np
import pytest

from atrip_gb300 import capi, synth

pytestmark = pytest.mark.gpu
NAMES = ("epsi", "epsa", "Tai", "Tabij", "Vabij", "Vijka", "Vabci")
J2 = ("Jijka", "Jabci")
# the two kernels' rounding of a cell's lower levels, as the comparison of
# their results on finite data has it
TOL = 2.0 ** -28


def _ctx(d, j=False):
    ctx = capi.Context(d["No"], d["Nv"], 0)
    for n in NAMES + (J2 if j else ()):
        ctx.upload(n, d[n])
    return ctx


def _same(x, y):
    np.testing.assert_array_equal(np.isnan(x), np.isnan(y))
    ok = ~np.isnan(y)
    if ok.any():
        assert np.max(np.abs(x - y)[ok]) <= TOL * np.max(np.abs(y)[ok])


@pytest.mark.parametrize("form,S,variant", [("split_f16", 2, 2), ("split_bf16", 2, 1),
                                            ("split_bf16", 3, 1), ("split_bf16", 4, 1)])
@pytest.mark.parametrize("tensor,value", [("Tabij", np.nan), ("Vabci", np.nan), ("Vijka", np.nan),
                                          ("Jabci", np.nan), ("Tabij", np.inf), ("Vabci", -np.inf)])
def test_not_finite(form, S, variant, tensor, value):
    j = tensor in J2
    d = synth.make_inputs(8, 40, 22, with_j=j)
    d[tensor][3, 4, 5, 6] = value
    n = 3000
    with _ctx(d, j) as ctx:
        kw = dict(form=form, slices=S, use_j=j, max_iterations=n - 1)
        ctx.run(**kw)
        e, ect = ctx.tuple_energies(0, n)
        ctx.set_tuning(split_variant=variant)
        ctx.run(**kw)
        f, fct = ctx.tuple_energies(0, n)
    assert np.isnan(fct).any()
    _same(e, f)
    _same(ect, fct)


@pytest.mark.parametrize("form,S", [("split_f16", 2), ("split_bf16", 3)])
def test_not_finite_in_a_batch(form, S):
    ds = [synth.make_inputs(8, 20, 23), synth.make_inputs(5, 17, 24)]
    ds[1]["Vabci"][3, 4, 5, 1] = np.nan
    ctxs = [_ctx(d) for d in ds]
    out = []
    with capi.Batch(ctxs) as b:
        for variant in (0, 2):
            b.set_tuning(split_variant=variant)
            b.run(form=form, slices=S, use_j=False)
            out.append([c.tuple_energies(0, synth.n_tuples(d["Nv"]))[0] for c, d in zip(ctxs, ds)])
    for c in ctxs:
        c.close()
    assert np.isnan(out[1][1]).any() and not np.isnan(out[1][0]).any()
    for x, y in zip(*out):
        _same(x, y)


# every digit product of level 1 of one sign: its sum passes 2^31 from
# K = 2 (Nv + No) = 1100 or so on.  T and V depend on their indices by the first
# digit: a W cell that is the same under all permutations has no energy.  Digits
# are multiples of 16, so every sum is exact in FP32, in either kernel
@pytest.mark.parametrize("No,Nv", [(2, 500), (2, 600), (3, 700)])
def test_coherent_digits_f16(No, Nv):
    torch = pytest.importorskip("torch")
    top, low = 1008, 1008 / 2048  # first and second digit
    x = (top + low) / 1024
    v = torch.arange(Nv, dtype=torch.float64, device="cuda").clamp(max=4)
    p = torch.arange(No, dtype=torch.float64, device="cuda")

    def const(n, value):
        return torch.full((n,), value, dtype=torch.float64, device="cuda")

    def tensor(t):  # column-major data of t[first index, ...]
        return t.permute(*reversed(range(t.dim()))).contiguous().ravel()

    with capi.Context(No, Nv, 0) as ctx:
        for k, t in (("epsi", const(No, -1.0)), ("epsa", const(Nv, 1.0)), ("Tai", const(Nv * No, 0.01)),
                     ("Vabij", const(Nv * Nv * No * No, 0.1)), ("Vijka", const(No ** 3 * Nv, -x))):
            torch.cuda.synchronize()
            ctx.upload(k, t)
        t = top + low - 16 * v[:, None, None, None] - 112 * p[:, None] - 208 * p
        t = tensor(t.expand(Nv, Nv, No, No) / 1024)
        torch.cuda.synchronize()
        ctx.upload("Tabij", t)
        t = top + low - 32 * v[None, :, None, None] - 160 * p
        t = tensor(t.expand(Nv, Nv, Nv, No) / 1024)
        torch.cuda.synchronize()
        ctx.upload("Vabci", t)
        ctx.run(form="split_f16", use_j=False, max_iterations=99)
        e, _ = ctx.tuple_energies(0, 100)
        ctx.set_tuning(split_variant=2)
        ctx.run(form="split_f16", use_j=False, max_iterations=99)
        f, _ = ctx.tuple_energies(0, 100)
    del t
    torch.cuda.empty_cache()
    _same(e, f)
