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
