"""Runs on a device that is nearly full: what fails says so, and what comes
after it works."""
import numpy as np
import pytest

from atrip_gb300 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
NAMES = ("epsi", "epsa", "Tai", "Tabij", "Vabij", "Vijka", "Vabci")
J2 = ("Jijka", "Jabci")
MB = 1 << 20


class full_device:
    """All of the device's free memory but `leave` bytes, while it lasts."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.block = torch.empty(max(0, free - self.leave), dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        del self.block
        torch.cuda.empty_cache()


def _ctx(d, j=False):
    ctx = capi.Context(d["No"], d["Nv"], 0)
    for n in NAMES + (J2 if j else ()):
        ctx.upload(n, d[n])
    return ctx


# W buffers of the transposed split kernel at No=40: 467 MB, 934 MB with (cT)
def test_split_run_after_a_failed_one():
    d = synth.make_inputs(40, 16, 31, with_j=True)
    with _ctx(d, True) as ctx:
        ctx.set_tuning(split_variant=2)
        ref = ctx.run(form="split_f16", use_j=False)
        with full_device(200 * MB):
            with pytest.raises(capi.AtripError) as err:
                ctx.run(form="split_f16", use_j=True)
            assert err.value.status == capi.ERR_OUT_OF_MEMORY
            again = ctx.run(form="split_f16", use_j=False)
        assert again.energy == ref.energy
        assert ctx.run(form="split_f16", use_j=True).energy == ref.energy


def _run64(ctx, n=200):
    ctx.run(form="fp64", use_j=False, max_iterations=n - 1)
    return ctx.tuple_energies(0, n)[0]


def _close(x, y, K):
    assert np.max(np.abs(x - y)) <= K * 2.0 ** -52 * np.max(np.abs(y))


# the slices of No=16/Nv=160 take about 2.5 GB; a second context of No=16/Nv=120
# needs 0.5 GB while V_pphp is uploaded
def test_another_context_takes_the_slices_memory():
    d, d2 = synth.make_inputs(16, 160, 32), synth.make_inputs(16, 120, 33)
    with _ctx(d) as ctx:
        e = _run64(ctx)
        with full_device(300 * MB):
            with _ctx(d2) as other:
                f = _run64(other)
            _close(_run64(ctx), e, 2 * 176)  # by whatever kernel there is memory for
        with _ctx(d2) as other:
            _close(f, _run64(other), 2 * 136)


# the DFMA kernel's workspace (155 MB or more at No=40) beside the slices
def test_tuned_run_takes_the_slices_memory():
    d = synth.make_inputs(40, 60, 34)
    with _ctx(d) as ctx:
        e = _run64(ctx)
        with full_device(50 * MB):
            ctx.set_tuning(fp64_tile_rows=64)
            _close(_run64(ctx), e, 2 * 100)


# FP16 slices of four systems (0.7 GB) beside their FP64 slices (2.5 GB)
def test_split_batch_takes_the_slices_memory():
    ds = [synth.make_inputs(16, 100 + k, 35 + k) for k in range(4)]
    opt = dict(use_j=False, max_iterations=499)
    out = []
    for leave in (100 * MB, 1 << 50):
        ctxs = [_ctx(d) for d in ds]
        with capi.Batch(ctxs) as b:
            e = b.run(form="fp64", **opt)
            with full_device(leave):
                out.append([r.energy for r in b.run(form="split_f16", **opt)])
            assert [r.energy for r in b.run(form="fp64", **opt)] == [r.energy for r in e]
        for c in ctxs:
            c.close()
    assert out[0] == out[1]


def test_trim_gives_the_slices_back():
    d = synth.make_inputs(16, 160, 32)
    with _ctx(d) as ctx:
        e = _run64(ctx)
        before = torch.cuda.mem_get_info()[0]
        ctx.trim()
        # V_pphp of 524 MB: slices of twice that and more
        assert torch.cuda.mem_get_info()[0] - before > 1000 * MB
        np.testing.assert_array_equal(_run64(ctx), e)
        ctx.trim()
        ctx.trim()


# (cT) slices that fit only in part are not kept: No=16/Nv=100, J_pphp in two
# FP16 slices 131 MB after J_hhhp's
def test_failed_ct_slices_leave_nothing_behind():
    d = synth.make_inputs(16, 100, 36, with_j=True)
    kw = dict(form="split_f16", max_iterations=99)
    with _ctx(d, True) as ctx:
        ctx.run(use_j=False, **kw)
        with full_device(96 * MB):
            free = []
            for _ in range(4):
                with pytest.raises(capi.AtripError) as err:
                    ctx.run(use_j=True, **kw)
                assert err.value.status == capi.ERR_OUT_OF_MEMORY
                free.append(torch.cuda.mem_get_info()[0])
        assert free[-1] == free[0]
        ref = ctx.run(use_j=True, **kw)
        assert np.isfinite(ref.ct_energy)


# a thread that runs FP64 ranges while another creates, uploads and closes a
# context for which there is room only without the first one's slices
def test_slices_are_taken_between_a_threads_runs():
    import threading
    d, d2 = synth.make_inputs(12, 110, 37), synth.make_inputs(16, 120, 38)
    bad, done = [], threading.Event()

    def runs(ctx, ref):
        try:
            for _ in range(300):
                _close(_run64(ctx, 100), ref, 2 * 122)
        except Exception as e:  # noqa: BLE001 - reported below
            bad.append(repr(e))
        done.set()

    with _ctx(d) as ctx:
        ref = _run64(ctx, 100)
        with full_device(400 * MB):
            t = threading.Thread(target=runs, args=(ctx, ref))
            t.start()
            made = 0
            while not done.is_set():
                try:
                    with _ctx(d2):
                        made += 1
                except capi.AtripError as e:  # the other one is in a call
                    if e.status != capi.ERR_OUT_OF_MEMORY:
                        bad.append(repr(e))
            t.join()
        assert not bad
        _close(_run64(ctx, 100), ref, 2 * 122)
