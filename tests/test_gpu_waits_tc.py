"""Bounded waits of the tensor-core kernel that the FP64 form and, by the engine's
choice, the split forms run on: as for the split kernels, a wait that runs out
(no tuple is ever published, nothing is copied or multiplied) ends the launch
with ATRIP_ERR_TIMEOUT and leaves the context usable."""
import pytest

from atrip_gb300 import capi, synth

pytestmark = pytest.mark.gpu
NAMES = ("epsi", "epsa", "Tai", "Tabij", "Vabij", "Vijka", "Vabci")


@pytest.mark.parametrize("form,slices,No,Nv,field", [
    ("fp64", 0, 8, 40, "real"), ("fp64", 0, 9, 30, "complex"), ("split_f16", 2, 8, 40, "real"),
    ("split_bf16", 3, 13, 30, "real"), ("split_bf16", 4, 40, 12, "real")])
def test_wait_runs_out_then_context_recovers(form, slices, No, Nv, field):
    d = synth.make_inputs(No, Nv, 3, field=field)
    with capi.Context(No, Nv, 0, field=field) as ctx:
        for n in NAMES:
            ctx.upload(n, d[n])
        kw = dict(form=form, slices=slices, use_j=False)
        ref = ctx.run(**kw)
        # ~10 ms limit (2e7 SM cycles)
        ctx.set_tuning(split_wait_kcycles=20000, split_test_unpublished=1)
        with pytest.raises(capi.AtripError) as err:
            ctx.run(**kw)
        assert err.value.status == capi.ERR_TIMEOUT
        assert "tensor-core kernel: a bounded wait" in str(err.value)
        ctx.set_tuning()
        assert ctx.run(**kw).energy == ref.energy
