"""FP64 form on the tensor cores (8-bit digit slices, exact sums) against the
DFMA kernel, which an explicit fp64_tile_rows selects, and the CPU oracle.

Both kernels round W like an FP64 dot product of K = 2 (Nv + No) terms: per
tuple they agree within K 2^-52 of the largest tuple energy.
"""
import numpy as np
import pytest

import oracle
from atrip_gb300 import capi, synth

pytestmark = pytest.mark.gpu
NAMES = ("epsi", "epsa", "Tai", "Tabij", "Vabij", "Vijka", "Vabci")
DFMA_LAUNCHES = 3  # the kernel and the two stages of the energy sum


def _ctx(d, j=False, field="real"):
    ctx = capi.Context(d["No"], d["Nv"], 0, field=field)
    for n in NAMES + (("Jijka", "Jabci") if j else ()):
        ctx.upload(n, d[n])
    return ctx


def _both(ctx, **kw):
    """(tensor-core result, its energies, DFMA energies) over one range."""
    r = ctx.run(form="fp64", **kw)
    t0, n = kw.get("first_iteration", 0), r.tuples_done
    e, ect = ctx.tuple_energies(t0, n)
    ctx.set_tuning(fp64_tile_rows=64)
    rd = ctx.run(form="fp64", **kw)
    assert rd.kernel_launches == DFMA_LAUNCHES
    d, dct = ctx.tuple_energies(t0, n)
    ctx.set_tuning()
    return r, (e, ect), (d, dct)


def _close(x, y, K):
    assert np.max(np.abs(x - y)) <= K * 2.0 ** -52 * np.max(np.abs(y))


# P = No rounded up to 8; N = 8 P of the widest MMA splits above 256; TMEM
# holds two accumulators up to No = 32; 128-row tiles end in No^2's remainder
@pytest.mark.parametrize("No,Nv,j", [
    (4, 80, False), (5, 66, True), (8, 40, True), (9, 47, False), (11, 64, False), (12, 65, True),
    (16, 33, False), (17, 33, True), (24, 30, False), (25, 21, False), (32, 18, True),
    (33, 20, False), (40, 24, True), (47, 16, False), (56, 14, False), (64, 12, False)])
def test_matches_dfma_and_oracle(No, Nv, j):
    d = synth.make_inputs(No, Nv, 11, with_j=j)
    n = min(synth.n_tuples(Nv), 700)
    with _ctx(d, j) as ctx:
        r, (e, ect), (f, fct) = _both(ctx, max_iterations=n - 1, use_j=j)
        assert r.kernel_launches > DFMA_LAUNCHES  # the slices were cut
        again = ctx.run(form="fp64", max_iterations=n - 1, use_j=j)
        assert again.energy == r.energy and again.kernel_launches == DFMA_LAUNCHES
        K = 2 * (Nv + No)
        _close(e, f, K)
        _close(ect, fct, K)
        pr = oracle.Problem(d)
        o = oracle.tuple_energies(pr, 0, 12)[0]
        assert np.max(np.abs(e[:12] - o)) <= K * 2.0 ** -52 * np.max(np.abs(f))


# complex: two column blocks of No rounded up to 8, products of K = 4 (Nv + No)
# real terms each; complex orbital energies
@pytest.mark.parametrize("No,Nv,j", [(5, 48, True), (8, 33, False), (9, 30, True), (13, 26, False),
                                     (17, 21, True), (24, 16, False), (32, 12, True)])
def test_complex_matches_dfma_and_oracle(No, Nv, j):
    d = synth.make_inputs(No, Nv, 12, with_j=j, field="complex", eps_imag=0.05)
    n = min(synth.n_tuples(Nv), 500)
    with _ctx(d, j, "complex") as ctx:
        r, (e, ect), (f, fct) = _both(ctx, max_iterations=n - 1, use_j=j, ijkabc=True)
        assert r.kernel_launches > DFMA_LAUNCHES
        K = 4 * (Nv + No)
        _close(e, f, K)
        _close(ect, fct, K)
        o = oracle.tuple_energies(oracle.Problem(d), 0, 8, ijkabc=True)[0]
        assert np.max(np.abs(e[:8] - o)) <= K * 2.0 ** -52 * np.max(np.abs(f))


# data the exact sums cannot hold runs on the DFMA kernel, with its result
@pytest.mark.parametrize("spoil", ["inf", "range", "constant"])
def test_data_rules(spoil):
    d = synth.make_inputs(8, 40, 13)
    if spoil == "inf":
        d["Vabci"][3, 4, 5, 6] = np.inf
    elif spoil == "range":
        d["Vabci"][:, 7] *= 2.0 ** -20
    else:  # every level sum coherent
        d["Tabij"][:] = 1.0 / 3.0
        d["Vabci"][:] = 1.0 / 3.0
    with _ctx(d) as ctx:
        r = ctx.run(form="fp64", max_iterations=199)
        e, _ = ctx.tuple_energies(0, 200)
        ctx.set_tuning(fp64_tile_rows=64)
        ctx.run(form="fp64", max_iterations=199)
        f, _ = ctx.tuple_energies(0, 200)
    np.testing.assert_array_equal(e, f)


# the no-allocation entry point's tensor-core kernel: tiles of 128 rows and
# their remainders, sums drained once and in pieces (2 (Nv + No) > 341), (cT);
# and data that sends it to its FP64-instruction kernel
@pytest.mark.parametrize("No,Nv,j,spoil", [(8, 40, True, False), (13, 33, False, False),
                                           (24, 26, True, False), (41, 18, False, False),
                                           (64, 12, False, False), (6, 170, False, False),
                                           (12, 40, False, True)])
def test_noalloc_tensor_cores(No, Nv, j, spoil):
    torch = pytest.importorskip("torch")
    import ctypes
    d = synth.make_inputs(No, Nv, 14, with_j=j)
    if spoil:
        d["Vabci"][:, 7] *= 2.0 ** -20
    names = NAMES + (("Jijka", "Jabci") if j else ())
    dev = {k: torch.from_numpy(np.ascontiguousarray(d[k].ravel(order="F"))).cuda() for k in names}
    n = min(synth.n_tuples(Nv), 3000 if No < 10 else 900 if No < 30 else 350)
    t0 = synth.n_tuples(Nv) - n
    out = torch.full((2 * n + 2,), float("nan"), dtype=torch.float64, device="cuda")
    ptrs = capi.DeviceInputs(*[dev[k].data_ptr() if k in dev else None for k in
                               NAMES + ("Jijka", "Jabci")])
    lib = capi.load()
    torch.cuda.synchronize()
    for _ in range(2):
        capi.check(lib.atrip_gpu_run_fp64_noalloc(
            No, Nv, ctypes.byref(ptrs), t0, t0 + n - 1, 0, 1, out.data_ptr() + 16,
            out.data_ptr() + 16 + 8 * n, out.data_ptr(), None))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    with _ctx(d, j) as ctx:
        ctx.set_tuning(fp64_tile_rows=64)
        r = ctx.run(form="fp64", first_iteration=t0, max_iterations=t0 + n - 1)
        e, ect = ctx.tuple_energies(t0, n)
    K = 2 * (Nv + No)
    _close(got[2:2 + n], e, K)
    _close(got[2 + n:], ect, K)
    assert abs(got[0] - r.energy) <= K * 2.0 ** -52 * np.sum(np.abs(e))


# split forms without launch parameters: the same digit products on the kernel
# of the FP64 form.  The kernels a variant selects round the levels above 0 to
# FP32 (2^-24 of a part 2^-8 of W or smaller, three groups, both factors of an
# energy): 2^-28 of the largest tuple energy.
@pytest.mark.parametrize("form,S", [("split_bf16", 2), ("split_bf16", 3), ("split_bf16", 4),
                                    ("split_f16", 2)])
@pytest.mark.parametrize("No,Nv,j", [(1, 9, False), (3, 17, True), (8, 40, False), (13, 64, True),
                                     (24, 30, True), (33, 17, False), (41, 65, False),
                                     (64, 10, True)])
def test_split_forms_match_split_kernels(No, Nv, j, form, S):
    d = synth.make_inputs(No, Nv, 15, with_j=j)
    n = min(synth.n_tuples(Nv), 600)
    with _ctx(d, j) as ctx:
        kw = dict(form=form, slices=S, use_j=j, max_iterations=n - 1, ijkabc=True)
        r = ctx.run(**kw)
        e, ect = ctx.tuple_energies(0, n)
        ctx.set_tuning(split_variant=2 if form == "split_f16" else 1)
        v = ctx.run(**kw)
        f, fct = ctx.tuple_energies(0, n)
    assert np.max(np.abs(e - f)) <= 2.0 ** -28 * np.max(np.abs(f))
    assert np.max(np.abs(ect - fct)) <= 2.0 ** -28 * np.max(np.abs(fct))
    assert abs(r.energy - v.energy) <= 2.0 ** -28 * np.sum(np.abs(f))
